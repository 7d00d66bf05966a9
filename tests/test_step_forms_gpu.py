"""The training step in the forms its sizes choose: rows read straight from the table, widths around a warp's pieces."""

import numpy as np
import pytest

from distributed_kge_poplar_b200 import capi
from helpers import assert_close, engine_settings, make_oracle, random_batch, random_state, read_rows, read_state, write_state
from oracle import step_oracle as so
from oracle.step_oracle import StepConfig

pytestmark = pytest.mark.gpu
RW = 64


def _config(score_fn, distance_fn, **sizes):
    return StepConfig(**{**dict(n_shard=1, n_entity=300, n_relation_type=12, embedding_size=16, entity_feature_size=0, batch_size=8, a2a_size=16,
                                score_fn=score_fn, distance_fn=distance_fn, gamma=6.0, loss_type="logsigmoid"), **sizes})


def _two_runs(cfg, seed, rtol, rel_rtol=None, dtype="float32", n_step=2, pad=3, feature_dtype=None, **extra):
    """Two program runs (plain launches, then graphs) against the oracle."""
    store = np.float32 if dtype == "float32" else np.float16
    state = random_state(cfg, seed, fp16_features=feature_dtype == "float16" or dtype == "float16", warm=True)
    state["entity_data"] = state["entity_data"].astype(store).astype(np.float32)
    engine = capi.CEngine(engine_settings(cfg, n_step=n_step, dtype=dtype, feature_dtype=feature_dtype, rw_batch=RW, **extra))
    write_state(engine, cfg, state, RW, dtype=store)
    oracle = make_oracle(cfg, state)
    for run in range(2):
        batch = random_batch(cfg, n_step, seed + 1 + run, pad=pad)
        want = oracle.train_step_loop(1e-3, batch)
        got = np.zeros(cfg.n_shard, np.float32)
        engine.run("train_step_loop", dict(learning_rate=np.full(cfg.n_shard, 1e-3, np.float32), loss=got, **batch))
        assert_close(got, want, rtol, f"loss of run {run}", atol_scale=0)
    want, d = oracle.get_state(), cfg.embedding_size
    got = read_state(engine, cfg, RW, cfg.n_shard) if dtype == "float32" else dict(entity_data=read_rows(engine, cfg, RW, cfg.n_shard, store).astype(np.float32))
    hidden = [engine.debug_fetch("hidden", s, cfg.n_remote * d).reshape(-1, d) for s in range(cfg.n_shard)]
    d_hidden = [engine.debug_fetch("d_hidden", s, cfg.n_remote * d).reshape(-1, d) for s in range(cfg.n_shard)]
    raw = [engine.debug_fetch("raw_score", s, cfg.batch_size * cfg.n_tail).reshape(cfg.batch_size, -1) for s in range(cfg.n_shard)]
    engine.close()
    for s in range(cfg.n_shard):
        assert_close(hidden[s], oracle.last["hidden"][s], rtol, f"hidden[{s}]")
        scores = cfg.gamma - raw[s] if cfg.score_fn in ("TransE", "RotatE", "TransH") else raw[s]
        assert_close(scores, oracle.last["scores"][s], rtol, f"scores[{s}]")
        if cfg.share_feature_networks and cfg.distance_fn != "L1":
            assert_close(d_hidden[s], oracle.last["d_feature_hidden"][s], rtol, f"d hidden[{s}]")
    assert_close(got["entity_data"][..., : 3 * d], want["entity_data"][..., : 3 * d], rtol, "rows")
    for key in set(got) & set(want) - {"entity_data", "step"}:
        assert_close(got[key], want[key], (rel_rtol if key.startswith("relation") else None) or rtol, key)


# the bounds of several steps of the other step tests: 1e-4, and 2e-3 where relation gradients pass through float16
@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L1"), ("TransE", "L2"), ("DistMult", "MatMul"), ("ComplEx", "MatMul"), ("RotatE", "L2")])
@pytest.mark.parametrize("d", [4, 36, 132, 516])
def test_rows_straight_from_the_table(score_fn, distance_fn, d):
    """Without features: a row of one piece, of a warp's pieces and a remainder, and of more than a lane keeps in flight."""
    _two_runs(_config(score_fn, distance_fn, embedding_size=d), seed=d, rtol=1e-4, rel_rtol=2e-3 if score_fn == "RotatE" else None)


def test_rows_straight_from_a_float16_table():
    # float16 rows: the bound of the other float16 tests
    _two_runs(_config("ComplEx", "MatMul", embedding_size=36, n_shard=2), seed=5, rtol=2e-2, dtype="float16")


@pytest.mark.parametrize("n_shard", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L1"), ("TransE", "L2"), ("DistMult", "MatMul"), ("RotatE", "L2"), ("TransH", "L1")])
def test_batches_of_any_size(score_fn, distance_fn, n_shard):
    """One launch for up to four shards, a fifth in one of its own, nine in three groups; batches and tails that fill no tile and no 16 bytes."""
    cfg = _config(score_fn, distance_fn, n_shard=n_shard, batch_size=7 * n_shard, a2a_size=9, n_relation_type=2 * n_shard, embedding_size=20, entity_feature_size=n_shard * 6,
                  loss_type="softmax", correction_weight=1.0)
    _two_runs(cfg, seed=n_shard, rtol=1e-4, rel_rtol=2e-3 if score_fn == "RotatE" else None, feature_dtype="float16" if n_shard % 2 else None)


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L1"), ("ComplEx", "MatMul"), ("TransH", "L1")])
@pytest.mark.parametrize("fused", ["1", "0"])
def test_shards_update_dense_parameters_together(monkeypatch, score_fn, distance_fn, fused):
    """Relation rows that no, one and all shards name; the Adam step in the row update and in a kernel of its own."""
    monkeypatch.setenv("KGE_FUSE_DENSE_UPDATE", fused)
    cfg = _config(score_fn, distance_fn, n_shard=4, batch_size=8, a2a_size=5, n_relation_type=40, learning_rate_modifiers={"relation_embedding": 0.5})
    _two_runs(cfg, seed=3, rtol=1e-4)


def test_separate_networks_of_four_shards():
    _two_runs(_config("TransE", "L2", n_shard=4, batch_size=12, a2a_size=7, embedding_size=36, entity_feature_size=12, share_feature_networks=False), seed=9, rtol=1e-4)


def test_groups_of_shards_run_side_by_side():
    """Sixteen small shards are four groups whose launches are too small to keep one another waiting: one after the other a step
    took 4.2 times the step of one group, side by side 1.8 times."""
    def ms_per_run(n_shard):
        cfg = _config("TransE", "L1", n_shard=n_shard, n_entity=1000, n_relation_type=16, embedding_size=8, entity_feature_size=16, batch_size=32, a2a_size=5)
        engine = capi.CEngine(engine_settings(cfg, n_step=10, rw_batch=RW))
        write_state(engine, cfg, random_state(cfg, 1), RW)
        run = dict(learning_rate=np.full(n_shard, 1e-3, np.float32), loss=np.zeros(n_shard, np.float32), **random_batch(cfg, 10, 2))
        times = []
        for _ in range(12):
            engine.run("train_step_loop", run)
            times.append(engine.last_run_stats()[0])
        engine.close()
        return min(times[2:])

    four, sixteen = ms_per_run(4), ms_per_run(16)
    assert sixteen < 3 * four, f"{sixteen:.3f} ms for sixteen shards, {four:.3f} ms for four"


def test_odd_widths_count_no_ties():
    """L1 gradients add a chunk up again where a difference is 0, which the missing neighbour of an odd row's last column must not
    look like: 63 columns take as long as 62, whose blocks and copies are the same, and not as long as all chunks twice."""
    def us_per_step(d):
        cfg = _config("TransE", "L1", n_entity=2000, embedding_size=d, batch_size=512, a2a_size=768)
        engine = capi.CEngine(engine_settings(cfg, n_step=20, rw_batch=RW))
        write_state(engine, cfg, random_state(cfg, 1), RW)
        run = dict(learning_rate=np.full(1, 1e-3, np.float32), loss=np.zeros(1, np.float32), **random_batch(cfg, 20, 2))
        times = []
        for _ in range(6):
            engine.set_kernel_timing(True)
            engine.run("train_step_loop", run)
            ms, launches = engine.kernel_times()["score_bwd"]
            times.append(1e3 * ms / launches)
        engine.close()
        return min(times[1:])

    odd, even = us_per_step(63), us_per_step(62)
    assert odd < 1.2 * even, f"{odd:.1f} us for 63 columns, {even:.1f} us for 62"


@pytest.mark.parametrize("fn", [capi.L1, capi.L2, capi.DOT], ids=["l1", "l2", "dot"])
@pytest.mark.parametrize("shape", [(1, 1, 4), (64, 33, 128), (65, 49, 132), (130, 700, 260), (200, 1500, 288), (64, 64, 516)])
def test_scores_in_blocks(fn, shape):
    """Blocks of 32, 48 and 64 columns with and without a remainder; one chunk of k, four, five, eight and more."""
    m, n, k = shape
    rng = np.random.RandomState(n)
    a, b = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(n, k)).astype(np.float32)
    b[-1] = a[0]
    a64, b64 = a.astype(np.float64), b.astype(np.float64)
    want = {capi.L1: so.l1_distance, capi.L2: so.l2_distance, capi.DOT: lambda x, y: x @ y.T}[fn](a64, b64)
    assert_close(capi.op_pairwise(fn, a, b), want, 1e-5, f"scores {shape}")


@pytest.mark.parametrize("score_fn,distance_fn", [("RotatE", "L2"), ("ComplEx", "MatMul")])
@pytest.mark.parametrize("batch,a2a", [(64, 1536), (70, 900), (1000, 150), (300, 2200)])
def test_score_gradients_of_lopsided_batches(score_fn, distance_fn, batch, a2a):
    """Many more tails than triples and the reverse: the two contractions' k ranges divided differently, with clusters whose
    last tile has no rows.  Sums of up to 2200 cancelling terms: the bound of the other long contractions, 5e-5, over two steps."""
    _two_runs(_config(score_fn, distance_fn, n_entity=4000, batch_size=batch, a2a_size=a2a, embedding_size=68, loss_type="softmax", correction_weight=1.0), seed=batch, rtol=1e-4,
              rel_rtol=2e-3 if score_fn == "RotatE" else None, n_step=1)


@pytest.mark.parametrize("loss_type,adversarial", [("softmax", 0.0), ("logsigmoid", 0.0), ("logsigmoid", 1.5)])
@pytest.mark.parametrize("a2a", [2, 255, 257, 1023, 1025, 2049, 4090])
def test_loss_rows_of_any_length(loss_type, adversarial, a2a):
    """One column and more per thread, up to the longest row, the last of a thread's there and not; 256 and 512 threads."""
    cfg = _config("DistMult", "MatMul", n_entity=4200, batch_size=4, a2a_size=a2a, embedding_size=8, loss_type=loss_type, negative_adversarial_scale=adversarial)
    _two_runs(cfg, seed=a2a, rtol=1e-4, n_step=1, pad=1 if a2a == 2 else 3)


@pytest.mark.parametrize("rows,n_best", [(2, 1), (330, 5), (700, 32), (700, 33), (5200, 20)])
@pytest.mark.parametrize("same", [False, True], ids=["different", "ties"])
def test_first_scan_of_a_ranking(rows, n_best, same):
    """Parts with fewer scores than a warp holds, one more and several times as many; lists of up to 32 keys and longer ones;
    equal scores, of which every one reaches the cut-off (ties go to the lower row)."""
    from test_predict_gpu import _clear, _predict

    cfg = _config("TransE", "L1", n_shard=2, n_entity=rows + 1, batch_size=2, a2a_size=2, embedding_size=8)
    state = random_state(cfg, rows)
    if same:
        state["entity_data"][..., :8] = state["entity_data"][:, 1:2, :8]
    n_best = min(n_best, rows)
    engine = capi.CEngine(engine_settings(cfg, rw_batch=RW, **{"execution.predict_hr_batch_size": 3, "execution.predict_n_best": n_best}))
    write_state(engine, cfg, state, RW)
    rng = np.random.RandomState(1)
    queries = np.stack([np.arange(6) % 2, 1 + rng.randint(rows, size=6), rng.randint(12, size=6)], axis=1)
    counts = np.array([rows, max(n_best, rows - 3)])
    got_idx, got_score = _predict(engine, cfg, queries, counts, 3, n_best)
    engine.close()
    want_idx, want_score = make_oracle(cfg, state).predict(queries, counts, n_best)
    assert_close(got_score, want_score, 1e-5, "ranking: scores")
    clear = np.ones_like(want_score, bool) if same or n_best == 1 else _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])


@pytest.mark.parametrize("shape", [(64, 37888, 36), (65, 18945, 64), (64, 37889, 36)])
def test_scores_in_tiles_of_both_widths(shape):
    """One wave of 128-column tiles, the same with ragged ones, and one tile more: two waves, so tiles of 96 columns."""
    test_scores_in_blocks(capi.L1, shape)


@pytest.mark.parametrize("score_fn,distance_fn", [("TransE", "L1"), ("ComplEx", "MatMul"), ("RotatE", "L2"), ("TransH", "L1")])
@pytest.mark.parametrize("d,dtype", [(4, "float32"), (6, "float32"), (38, "float16"), (132, "float16")])
def test_ranked_queries_straight_from_the_table(score_fn, distance_fn, d, dtype):
    """Five shards without features: queries of four shards in a launch and the fifth by itself; 16-byte rows and others."""
    from test_predict_gpu import _clear, _predict

    store = np.dtype(dtype).type
    cfg = _config(score_fn, distance_fn, n_shard=5, n_entity=90, batch_size=10, a2a_size=4, n_relation_type=10, embedding_size=d)
    state = random_state(cfg, d)
    state["entity_data"] = state["entity_data"].astype(store).astype(np.float32)
    engine = capi.CEngine(engine_settings(cfg, rw_batch=RW, dtype=dtype, **{"execution.predict_hr_batch_size": 3}))
    write_state(engine, cfg, state, RW, dtype=store)
    rng = np.random.RandomState(1)
    queries = np.stack([np.arange(15) % 5, 1 + rng.randint(89, size=15), rng.randint(10, size=15)], axis=1)
    got_idx, got_score = _predict(engine, cfg, queries, np.full(5, 89), 3, 5)
    engine.close()
    want_idx, want_score = make_oracle(cfg, state).predict(queries, np.full(5, 89), 5)
    assert_close(got_score, want_score, 1e-5, "ranking: scores")
    clear = _clear(want_score)
    np.testing.assert_array_equal(got_idx[clear], want_idx[clear])


def _product_plus(a, x, y):
    """a x + y in float32 with one rounding, as an FMA gives it: the product is exact in float64, the sum is rounded to odd there,
    which float32's rounding of it cannot be misled by."""
    p, y = np.asarray(a, np.float32).astype(np.float64) * np.asarray(x, np.float64), np.asarray(y, np.float64)
    total = p + y
    back = total - p
    error = (p - (total - back)) + (y - back)
    even = (total.view(np.int64) & 1) == 0
    return np.where((error != 0) & even, np.nextafter(total, np.where(error > 0, np.inf, -np.inf)), total).astype(np.float32)


def _product(a, b):
    return np.float32(a) * np.float32(b)


@pytest.mark.parametrize("d,features,mlp", [(6, 0, 0), (16, 0, 0), (16, 12, 0), (16, 12, 8)], ids=["odd rows", "table rows", "gathered rows", "mlp"])
def test_row_moments_round_alike(d, features, mlp):
    """Every form of the row update rounds the moments' old part and not the gradient's: the bits of that sum."""
    cfg = _config("TransE", "L1", embedding_size=d, entity_feature_size=features, feature_mlp_size=mlp, loss_type="softmax", correction_weight=1.0)
    state = random_state(cfg, d, warm=True)
    batch = random_batch(cfg, 1, 3, pad=3)

    def step(cfg, state):
        engine = capi.CEngine(engine_settings(cfg, rw_batch=RW))
        write_state(engine, cfg, state, RW)
        engine.run("train_step_loop", dict(learning_rate=np.full(1, 1e-3, np.float32), loss=np.zeros(1, np.float32), **batch))
        out = engine.debug_fetch("d_hidden", 0, cfg.n_remote * d).reshape(-1, d), read_rows(engine, cfg, RW, 1, np.float32)[0]
        engine.close()
        return out

    if mlp:  # with a last layer of zeros the hidden rows are the values and nothing passes back: the gradients of the model without features
        state["mlp_down_projection"][:] = 0
        bare = {k: v for k, v in state.items() if "projection" not in k}
        grad, _ = step(_config("TransE", "L1", embedding_size=d, loss_type="softmax", correction_weight=1.0), dict(bare, entity_data=state["entity_data"][..., : 3 * d]))
        _, got = step(cfg, state)
    else:
        grad, got = step(cfg, state)
    remote = batch["remote"][0, 0]
    rows, slots = np.unique(remote, return_index=True)
    rows, slots = rows[rows > 0], slots[rows > 0]
    g, old = grad[slots], state["entity_data"][0][rows]
    one_m, one_v = np.float32(1) - np.float32(cfg.adam_beta_m), np.float32(1) - np.float32(cfg.adam_beta_v)
    np.testing.assert_array_equal(got[rows, d : 2 * d], _product_plus(one_m, g, _product(cfg.adam_beta_m, old[:, d : 2 * d])))
    root = old[:, 2 * d : 3 * d]
    want_v = _product_plus(_product(one_v, g), g, _product(cfg.adam_beta_v, _product(root, root)))
    np.testing.assert_array_equal(got[rows, 2 * d : 3 * d], np.sqrt(want_v))


@pytest.mark.parametrize("form", ["fused", "of its own", "separate kernels"])
def test_dense_moments_round_alike(monkeypatch, form):
    """Every form of the dense update rounds the gradient's part of the moments and not the old one's: the bits of that sum, for
    the projection (a contraction's epilogue or k_dense_update) and for the relations (the row update or k_dense_update)."""
    monkeypatch.setenv("KGE_FUSE_DENSE_UPDATE", "1" if form == "fused" else "0")
    d = 10 if form == "separate kernels" else 16
    cfg = _config("TransE", "L2", embedding_size=d, entity_feature_size=12, n_relation_type=12, batch_size=8, loss_type="softmax", correction_weight=1.0)
    state = random_state(cfg, d, warm=True)
    engine = capi.CEngine(engine_settings(cfg, rw_batch=RW))
    write_state(engine, cfg, state, RW)
    batch = random_batch(cfg, 1, 3, pad=3)
    batch["relation"][:] = np.arange(8)  # a triple per relation: no order of a sum to agree on
    engine.run("train_step_loop", dict(learning_rate=np.full(1, 1e-3, np.float32), loss=np.zeros(1, np.float32), **batch))
    grads = engine.debug_fetch("dense_grad", 0, 1 << 12)
    got = read_state(engine, cfg, RW, 1)
    engine.close()
    one_m, one_v = np.float32(1) - np.float32(cfg.adam_beta_m), np.float32(1) - np.float32(cfg.adam_beta_v)
    for name, g in (("relation_embedding", grads[: 12 * d].reshape(12, d)), ("feature_projection", grads[12 * d :].reshape(12, d))):
        m, v = state[name + "/adam_m"], state[name + "/adam_v"]
        np.testing.assert_array_equal(got[name + "/adam_m"], _product_plus(cfg.adam_beta_m, m, _product(one_m, g)), err_msg=name)
        np.testing.assert_array_equal(got[name + "/adam_v"], _product_plus(cfg.adam_beta_v, v, _product(_product(one_v, g), g)), err_msg=name)
