"""Calls of the CUDA runtime that fail, made to fail on the host: a preloaded library answers the n-th call of a function
with an error code and passes every other call on.  No kernel is disturbed."""

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

SHIM = r"""
#include <dlfcn.h>
#include <stdio.h>
#include <stdlib.h>
static void *runtime(const char *name) { return dlsym(dlopen("libcudart.so.12", RTLD_LAZY | RTLD_NOLOAD), name); }
static int due(const char *variable, int *calls) {  /* FAIL_<function>="n": the n-th call and all later ones, "n!": that one */
    const char *at = getenv(variable);
    if (!at) return 0;
    const int n = atoi(at);
    ++*calls;
    return at[1] == '!' ? *calls == n : *calls >= n;
}
int cudaGraphInstantiate(void **exec, void *graph, unsigned long long flags) {
    static int calls;
    if (due("FAIL_cudaGraphInstantiate", &calls)) return 2; /* out of memory */
    return ((int (*)(void **, void *, unsigned long long))runtime("cudaGraphInstantiate"))(exec, graph, flags);
}
int cudaGraphLaunch(void *exec, void *stream) {
    static int calls;
    if (due("FAIL_cudaGraphLaunch", &calls)) return 2;
    return ((int (*)(void *, void *))runtime("cudaGraphLaunch"))(exec, stream);
}
int cudaEventRecord(void *event, void *stream) {
    static int calls;
    if (due("FAIL_cudaEventRecord", &calls)) return 2;
    return ((int (*)(void *, void *))runtime("cudaEventRecord"))(event, stream);
}
int cudaHostAlloc(void **p, size_t bytes, unsigned flags) {
    if (getenv("SHOW_cudaHostAlloc")) puts("cudaHostAlloc"), fflush(stdout);
    return ((int (*)(void **, size_t, unsigned))runtime("cudaHostAlloc"))(p, bytes, flags);
}
int cudaEventElapsedTime(float *ms, void *begin, void *end) {
    static int calls;
    if (due("FAIL_cudaEventElapsedTime", &calls)) return 600; /* not ready */
    return ((int (*)(float *, void *, void *))runtime("cudaEventElapsedTime"))(ms, begin, end);
}
"""

PRELUDE = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
import numpy as np
from distributed_kge_poplar_b200 import capi
from helpers import read_state
from test_engine_gpu import CASES, RW, _build, _run_engine
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    folder = tmp_path_factory.mktemp("shim")
    (folder / "shim.c").write_text(SHIM)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(folder / "shim.c"), "-o", str(folder / "shim.so"), "-ldl"], check=True)
    return folder / "shim.so"


def _run(shim, body, **fail):
    env = dict(os.environ, LD_PRELOAD=str(shim), **{f"FAIL_{name}": value for name, value in fail.items()})
    script = PRELUDE.format(root=str(ROOT), tests=str(ROOT / "tests")) + body
    done = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout[-2000:] + done.stderr[-2000:]
    return done.stdout


def test_a_failing_event_read_is_an_error_code(shim):
    """An exception that left the C entry would end the process."""
    out = _run(shim, """
cfg, _, engine, batch = _build(CASES["config1_transe_l1"])
_run_engine(engine, cfg, batch, 1e-3)
try:
    engine.last_run_stats()
    print("no error")
except RuntimeError as e:
    print("raised", e)
assert engine.last_run_stats()[0] > 0
""", cudaEventElapsedTime="1!")
    assert out.startswith("raised") and "cudaEventElapsedTime" in out


def test_a_graph_that_finds_no_memory_leaves_the_run_whole(shim):
    """The second graph of a run cannot be made: its steps go out as plain launches, and later runs as graphs again."""
    _run(shim, """
case = CASES["config1_transe_l1"]
cfg, _, engine, batch = _build(case, n_step=6, warm=True)
_, _, plain, _ = _build(case, n_step=6, warm=True, cuda_graph=False)
for run in range(4):
    got, want = _run_engine(engine, cfg, batch, 1e-3), _run_engine(plain, cfg, batch, 1e-3)
    np.testing.assert_array_equal(got, want)
    assert engine.last_run_stats()[1] == plain.last_run_stats()[1], "launches"
a, b = (read_state(e, cfg, RW, cfg.n_shard) for e in (engine, plain))
for name in a:
    np.testing.assert_array_equal(a[name], b[name], err_msg=name)
""", cudaGraphInstantiate="2!")


def test_a_run_that_fails_half_way_makes_the_engine_unusable(shim):
    """The first of a run's graphs has moved the rows when the second cannot be launched."""
    _run(shim, """
cfg, _, engine, batch = _build(CASES["config1_transe_l1"], n_step=6, warm=True)
for run in range(3):
    try:
        _run_engine(engine, cfg, batch, 1e-3)
    except RuntimeError as e:
        assert "cudaGraphLaunch" in str(e), e
        break
else:
    raise SystemExit("no launch failed")
try:
    _run_engine(engine, cfg, batch, 1e-3)
except RuntimeError as e:
    assert "must be rebuilt" in str(e), e
else:
    raise SystemExit("the engine trains on")
""", cudaGraphLaunch="2!")


@pytest.mark.parametrize("command", ["read_entity_range", "read"])
def test_blocks_of_a_failed_transfer_are_not_lent_again(shim, command):
    """The transfer into the pinned block is under way when the event behind it fails: the block is freed, and the next
    transfers take others, and in the end a new one."""
    out = _run(shim, f"""
import os
cfg, state, engine, batch = _build(CASES["config1_transe_l1"])
rows = np.zeros((cfg.n_shard, 300, cfg.row_size), np.float32)
value = np.zeros((cfg.n_relation_type, cfg.embedding_size), np.float32)
arrays, name = (dict(row_range=np.array([1, 300], np.uint32), read_data=rows), None) if {command!r} != "read" else (dict(value=value), "relation_embedding")
engine.run({command!r}, arrays, name=name)
os.environ["SHOW_cudaHostAlloc"] = "1"
print("again", flush=True)
engine.run({command!r}, arrays, name=name)
os.environ["FAIL_cudaEventRecord"] = "1"
for block in range(4):  # as many as the pool keeps
    try:
        engine.run({command!r}, arrays, name=name)
        raise SystemExit("nothing failed")
    except RuntimeError:
        pass
print("failed", flush=True)
del os.environ["FAIL_cudaEventRecord"]
engine.run({command!r}, arrays, name=name)
np.testing.assert_array_equal(rows[..., : cfg.embedding_size] if name is None else value,
                              state["entity_data"][:, 1:301, : cfg.embedding_size] if name is None else state[name])
""")
    assert out.split()[0] == "again" and out.split()[-2:] == ["failed", "cudaHostAlloc"]
