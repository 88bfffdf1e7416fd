"""GPU tests of the autotuner on samples that the default answers with a warp per query, and of cache
entries made for other kernels."""
import numpy as np
import pytest

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return t


def _time(torch, f):
    t = []
    for _ in range(25):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b))
    return sorted(t[3:])[8]


def test_not_slower_than_the_default(torch):
    """4,096 queries: the best named variant takes several times the default's time."""
    V, F = W.uv_sphere(64, 32)
    Q = torch.from_numpy(W.box_queries(V, 4096, np.random.default_rng(0))).cuda()
    r = fwn.autotune(V, F, Q)
    tuned, default = fwn.FastWindingNumber(V, F, **r["config"]), fwn.FastWindingNumber(V, F)
    assert _time(torch, lambda: tuned.query(Q)) <= 2.0 * _time(torch, lambda: default.query(Q))


def test_forest_not_slower_than_the_default(torch):
    fo = W.batched_forest_workload(n_meshes=4, seed=6, f_lo=500, f_hi=4000, q_lo=500, q_hi=4000)
    r = fwn.autotune_forest(fo.V, fo.voff, fo.F, fo.foff, fo.Q, fo.qoff)
    Q = torch.from_numpy(fo.Q).cuda()
    tuned, default = (fwn.Forest(fo.V, fo.voff, fo.F, fo.foff, **c) for c in (r["config"], {}))
    assert _time(torch, lambda: tuned.query_forest(Q, fo.qoff)) <= \
        2.0 * _time(torch, lambda: default.query_forest(Q, fo.qoff))


def test_entries_of_other_kernels_are_not_used(torch, tmp_path):
    wl = W.displaced_icosphere_workload(nu=12, n_queries=2000)
    cache = tmp_path / "tune.txt"
    fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))
    key, rest = cache.read_text().split(" ", 1)
    cache.write_text(f"t2|{key.split('|', 1)[1]} {rest}")
    assert fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))["from_cache"] == 0
    assert fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))["from_cache"] == 1
