"""GPU test of the autotuner on cache entries made for other kernels."""
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


def test_entries_of_other_kernels_are_not_used(torch, tmp_path):
    wl = W.displaced_icosphere_workload(nu=12, n_queries=2000)
    cache = tmp_path / "tune.txt"
    fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))
    key, rest = cache.read_text().split(" ", 1)
    cache.write_text(f"t2|{key.split('|', 1)[1]} {rest}")
    assert fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))["from_cache"] == 0
    assert fwn.autotune(wl.V, wl.F, wl.Q, cache_path=str(cache))["from_cache"] == 1
