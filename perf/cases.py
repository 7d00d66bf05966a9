"""The work whose speed is followed: program runs of the training step, ranking, and moving the table in and out.

Every case goes through the host interface (``distributed_kge_poplar_b200.poplar_kge.Engine``) as a driver
script does, on one GPU that holds all shards of the model.  Sizes are those of the repository's presets,
benchmark and tests, with tables cut down so that three engines fit a GPU; tables beyond 100 000 rows are far
larger than the L2 cache.  Entity popularity is Zipf(1.1) and relation popularity Zipf(1.3), as in real graphs.
"""

import math

import numpy as np

from distributed_kge_poplar_b200 import poplar_kge as kge


def _case(do, **options):
    """A case with the defaults of the settings tree: plain TransE-L2 rows in float32, one shard."""
    case = dict(do=do, score_fn="TransE", distance_fn="L2", loss="logsigmoid", adversarial=0.0, gamma=10.0, n_shard=1,
                rows=90, relations=12, d=8, features=0, batch=0, a2a=0, steps=1, dtype="float32", feature_dtype="float32",
                bf16_values=False, zipf=True, queries=0, n_best=10, rw=128)
    assert set(options) - {"name"} <= set(case)
    case.update(options)
    return case


def listed():
    return [
        # The demo preset's program run: a handful of triples, where launches and host work are everything.
        _case("train", name="demo", distance_fn="L1", gamma=2.0, n_shard=2, rows=90, relations=12, d=8, features=6, batch=6, a2a=5,
              steps=5, rw=50),
        # A single step on a small graph in four shards (10 000 entities), as a script that looks at every step runs it.
        _case("train", name="tiny_l1_step", distance_fn="L1", n_shard=4, rows=2501, relations=32, d=64, batch=256, a2a=80),
        # The headline workload: TransE-L2 on the WikiKG90Mv2 shape, 100 steps per program run, text features.
        _case("train", name="transe_l2_features", loss="softmax", rows=2_500_001, relations=1387, d=256, features=768, batch=512, a2a=768,
              steps=100, feature_dtype="float16"),
        # The same graph with two of its shards on one GPU: half the tails come from the other shard.
        _case("train", name="transe_l2_two_shards", loss="softmax", n_shard=2, rows=1_000_001, relations=1388, d=256, features=768,
              batch=512, a2a=384, steps=20, feature_dtype="float16"),
        # Wide bf16 embeddings with dot-product scores, uniform ids, no features.
        _case("train", name="distmult_bf16", distance_fn="MatMul", rows=3_750_001, relations=1000, d=512, batch=1024, a2a=2048, steps=20,
              bf16_values=True, zipf=False),
        # Batches drawn on the device, ComplEx with the sampled softmax.
        _case("sampled", name="complex_sampled", score_fn="ComplEx", distance_fn="MatMul", loss="softmax", rows=1_000_001, relations=1000,
              d=400, batch=768, a2a=1536, steps=50),
        # The published submission's model: RotatE-L2 with self-adversarial weights on fp16 rows, 1536 tails per shard.
        _case("train", name="rotate_l2_fp16", score_fn="RotatE", adversarial=4.0, rows=1_000_001, relations=1387, d=256, features=768,
              batch=256, a2a=1536, steps=50, dtype="float16", feature_dtype="float16"),
        # A graph of 2.5 million entities without features in four shards, TransE-L1 on fp16 rows.
        _case("train", name="transe_l1_fp16", distance_fn="L1", n_shard=4, rows=625_152, relations=536, d=100, batch=256, a2a=128,
              steps=20, dtype="float16", feature_dtype="float16"),
        # The score function with a hyperplane per relation.
        _case("train", name="transh", score_fn="TransH", distance_fn="L1", loss="softmax", rows=500_001, relations=1387, d=128, batch=512,
              a2a=768, steps=10),
        # Ranking all rows of a shard for 1250 queries: the large end of evaluation.
        _case("rank", name="rank_l2_features", rows=2_500_001, relations=1387, d=256, features=768, feature_dtype="float16", queries=1250,
              n_best=100),
        # Ranking by L1 distance over four shards for a small set of queries, as between two training intervals.
        _case("rank", name="rank_l1_fp16", distance_fn="L1", n_shard=4, rows=40_001, relations=536, d=100, dtype="float16",
              feature_dtype="float16", queries=32, n_best=10),
        # Bringing a dataset's features into a fresh table in chunks and reading whole rows back.
        _case("stream", name="stream_rows", rows=20_001, relations=64, d=256, features=768, feature_dtype="float16", rw=512),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _size(rng, low, high, multiple):
    """Mostly a multiple of `multiple`, one time in four any whole number: both are met in practice."""
    n = _log_int(rng, low, high)
    return n if rng.random() < 0.25 else max(multiple, n // multiple * multiple)


def draw(rng):
    do = rng.choice(["train", "train", "train", "train", "train", "sampled", "rank", "rank", "stream"])
    n_shard = rng.choice([1, 1, 2, 4])
    score_fn = rng.choice(["TransE", "TransE", "DistMult", "ComplEx", "RotatE", "TransH"])
    if score_fn in ("DistMult", "ComplEx"):
        distance_fn = "MatMul"
    elif score_fn == "TransH":
        distance_fn = "L1"
    else:
        distance_fn = rng.choice(["L1", "L2"])
    dtype = rng.choice(["float32", "float32", "float16"])
    d = 2 * _size(rng, 16, 128 if distance_fn == "L1" else 256, 8)
    features = 0 if distance_fn == "L1" or rng.random() < 0.5 else n_shard * _log_int(rng, 32 // n_shard, 768 // n_shard)
    case = _case(do, score_fn=score_fn, distance_fn=distance_fn, n_shard=n_shard, loss=rng.choice(["logsigmoid", "softmax"]),
                 relations=n_shard * _log_int(rng, 4, 1400 // n_shard), d=d, features=features, dtype=dtype,
                 feature_dtype="float16" if dtype == "float16" or rng.random() < 0.5 else "float32")
    if do == "stream":
        case.update(rows=_log_int(rng, 1000, 20_000) // n_shard + 1, rw=_log_int(rng, 64, 1024))
        return case
    case.update(rows=_log_int(rng, 2000, 1_000_000 if do != "rank" else 400_000 if distance_fn != "L1" else 80_000) // n_shard + 1)
    if do == "rank":
        case.update(queries=_size(rng, 8, 512 if distance_fn != "L1" else 64, 8), n_best=rng.choice([10, 20, 50, 100]))
        return case
    pairs = _size(rng, 16, 512 // n_shard, 4)  # positives per pair of shards
    case.update(batch=pairs * n_shard, a2a=pairs + _size(rng, 8, max(16, 1024 // n_shard), 4),
                steps=_log_int(rng, 1, 50 if score_fn != "TransH" else 10),
                adversarial=1.0 if case["loss"] == "logsigmoid" and rng.random() < 0.3 else 0.0,
                bf16_values=dtype == "float32" and distance_fn == "MatMul" and rng.random() < 0.5)
    return case


def _settings(case, seed):
    s = kge.Settings.create_demo()
    m, d, t, e = s.model, s.data, s.training, s.execution
    s.seed = m.seed = d.seed = seed
    m.score_fn, m.distance_fn, m.n_shard, m.n_entity = case["score_fn"], case["distance_fn"], case["n_shard"], case["rows"]
    m.n_relation_type, m.embedding_size, m.entity_feature_size = case["relations"], case["d"], case["features"]
    m.gamma, m.negative_adversarial_scale = case["gamma"], case["adversarial"]
    # a standard deviation (init_scale / d) with which distances are about gamma and products about one, as in a trained model
    if case["distance_fn"] == "L2":
        m.init_scale = case["d"] * case["gamma"] / math.sqrt(3 * case["d"])
    elif case["distance_fn"] == "L1":
        m.init_scale = case["gamma"] / 1.4
    else:
        m.init_scale = case["d"] * (2 / math.sqrt(case["d"])) ** (1 / 3)
    d.batch_size, d.a2a_size = case["batch"] or 256, case["a2a"] or 512 // case["n_shard"]
    t.loss = kge.SoftmaxLoss(correction_weight=1.0) if case["loss"] == "softmax" else kge.LogSigmoidLoss()
    t.learning_rate = 1e-4  # well into a decaying schedule
    e.dtype, e.feature_dtype, e.train_steps_per_program_run = case["dtype"], case["feature_dtype"], case["steps"]
    e.rw_batch_size, e.predict_n_best = min(case["rw"], case["rows"]), min(case["n_best"], case["rows"] - 1)
    e.predict_hr_batch_size = max(1, case["queries"])
    if case["bf16_values"]:
        e.value_dtype = "bfloat16"  # an optional setting of the engine that the tree does not list
    return s.prepare()


def _ids(rng, case, limit, size, alpha):
    """Ranks below `limit`, most frequent first: P(k) ~ (k + 1)^-alpha, or uniform."""
    u = rng.random_sample(size)
    if not case["zipf"]:
        return (u * limit).astype(np.int64)
    return np.minimum(((limit ** (1 - alpha) - 1) * u + 1) ** (1 / (1 - alpha)) - 1, limit - 1).astype(np.int64)


def _tail_ids(rng, case, limit, size):
    """As _ids, with other entities in front: those that are often tails are not those that are often heads."""
    return (_ids(rng, case, limit, size, 1.1) + limit // 2) % limit


def _batch(case, rng):
    """The index streams of one program run, laid out as the dataset's sampler does: positives bucketed by (head shard, tail
    shard), negatives shared by a shard's batch, every row gathered once, padding rows last."""
    n, S, B, a2a, rows = case["n_shard"], case["steps"], case["batch"], case["a2a"], case["rows"]
    pos = B // n
    head = (1 + _ids(rng, case, rows - 1, (n, S, n * pos), 1.1)).astype(np.uint32)
    tail = (1 + _tail_ids(rng, case, rows - 1, (n, S, n, pos))).astype(np.uint32)  # [head shard, step, tail shard, positive]
    negative = rng.randint(1, rows, size=(n, S, n, a2a - pos)).astype(np.uint32)  # [serving shard, step, asking shard, ...]
    served = np.concatenate([tail.transpose(2, 1, 0, 3), negative], axis=3)  # [serving shard, step, asking shard, a2a]
    wanted = np.concatenate([head, served.reshape(n, S, n * a2a)], axis=2)
    remote, lookup = np.zeros_like(wanted), np.zeros_like(wanted)
    for shard in range(n):
        for step in range(S):
            unique, inverse = np.unique(wanted[shard, step], return_inverse=True)
            remote[shard, step, : unique.size] = unique
            lookup[shard, step] = inverse
    label = (np.arange(n)[:, None] * a2a + np.arange(pos)).reshape(-1).astype(np.uint32)
    return kge.Batch(remote=remote, a2a=np.ascontiguousarray(lookup[:, :, B:]).reshape(n, S, n, a2a), head=np.ascontiguousarray(lookup[:, :, :B]),
                     relation=_ids(rng, case, case["relations"], (n, S, B), 1.3).astype(np.uint32),
                     tail=np.ascontiguousarray(np.broadcast_to(label, (n, S, B))))


def prepare(case, seed):
    rng = np.random.RandomState(seed % (1 << 32))
    n, rows = case["n_shard"], case["rows"]
    settings = _settings(case, seed % (1 << 30))
    engine = kge.Engine(settings, np.full(n, rows - 1, np.int64))
    state = dict(do=case["do"], engine=engine)
    if case["do"] == "stream":
        state["features"] = rng.standard_normal((n, rows, case["features"])).astype(np.float16).astype(np.float32)
        return state
    engine.initialise_variables()
    engine.engine.run("initialise_entities", {})
    engine.uninitialized_entity_data[:] = False
    if case["do"] == "train":
        state["batch"] = _batch(case, rng)
    elif case["do"] == "sampled":
        count, entities = 200_000, n * (rows - 1)
        hrt = np.stack([_ids(rng, case, entities, count, 1.1), _ids(rng, case, case["relations"], count, 1.3),
                        _tail_ids(rng, case, entities, count)], axis=1)
        ids = np.arange(entities)
        engine.load_triples(hrt, ids % n, ids // n + 1)
    else:
        if case["features"]:
            # the projection of a trained model: its spectrum falls off, so that candidates are spread out
            rank = min(32, case["features"], case["d"])
            left, right = rng.standard_normal((case["features"], rank)), rng.standard_normal((rank, case["d"]))
            scale = engine.init_scale / math.sqrt(case["features"] * rank)
            engine.write_variable("feature_projection", (2 * scale * left @ right).astype(np.float32))
        q = case["queries"] * n
        state["queries"] = np.stack([np.arange(q) % n, 1 + _ids(rng, case, rows - 1, q, 1.1), _ids(rng, case, case["relations"], q, 1.3)],
                                    axis=1).astype(np.uint32)
    return state


def run(state):
    engine = state["engine"]
    if state["do"] == "rank":
        best = engine.predict(state["queries"])
        return dict(score=best.score, shard_idx=best.shard_idx)
    if state["do"] == "stream":
        engine.initialise_all(state["features"])
        return engine.read_entity_all()
    loss, _ = engine.train_step_loop(state["batch"]) if state["do"] == "train" else engine.train_step_loop_sampled(1)
    # what a training loop looks at between program runs: the relations, and the rows of the most frequent entities
    return dict(loss=loss, relation=engine.read_variable("relation_embedding"), rows=engine.read_entity(0))


def work(case):
    n, S, B, D, F = case["n_shard"], case["steps"], case["batch"], case["d"], case["features"]
    state, feature = 4 if case["dtype"] == "float32" else 2, 4 if case["feature_dtype"] == "float32" else 2
    value = 2 if case["bf16_values"] else state
    if case["do"] == "stream":
        count = n * case["rows"]
        return dict(bytes=count * (4 * F + state * (3 * D + F)) + 2 * count * (D * (value + 2 * state) + F * feature), flops=0)
    per_pair = 2 if case["distance_fn"] == "MatMul" else 3
    if case["do"] == "rank":
        count, asked = n * (case["rows"] - 1), n * case["queries"]
        return dict(bytes=count * (D * value + F * feature) + asked * D * 4 + asked * case["n_best"] * 12,
                    flops=count * (2 * F * D + asked * D * per_pair))
    T = n * case["a2a"]
    R = B + T
    dense = (case["relations"] * (2 if case["score_fn"] == "TransH" else 1) + F) * D * 4
    step_bytes = n * R * (2 * D * (value + 2 * state) + F * feature) + 6 * dense
    step_flops = n * (per_pair * B * T * D + 4 * B * T * D + 4 * R * F * D)
    return dict(bytes=S * step_bytes, flops=S * step_flops)


def tolerance(case):
    if case["do"] == "stream":
        return "exact"
    if case["do"] == "rank":
        return dict(rel=1e-5, differ=0.01)  # fp32 sums; two candidates whose scores agree to rounding may change places
    # Sums in fp32 agree to about 1e-6 after a step; a program run's later steps and Adam's first step of a row, whose size
    # does not depend on the gradient's, carry that on, and an L1 gradient is a sum of signs, one of which may flip.
    if case["bf16_values"]:
        return dict(rel=1e-2, max=0.2)
    if case["dtype"] == "float16" or case["distance_fn"] == "L1":
        return dict(rel=1e-3, max=0.05)
    return dict(rel=1e-4, max=0.05)
