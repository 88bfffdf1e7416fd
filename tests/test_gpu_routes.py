"""GPU tests of which walk a batch takes."""
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


def _scratch(torch, f):
    """Bytes of query scratch that a call takes: the group walk's sort needs 16 per query, a warp per
    query none."""
    used = fwn.scratch_pool_stats(reset_high=True)["used"]
    res = f()
    torch.cuda.synchronize()
    return fwn.scratch_pool_stats()["used_high"] - used, res


@pytest.mark.parametrize("by_config", [False, True])
def test_explicit_warp_schedule_is_the_group_walk(torch, by_config):
    n = 20_000
    wl = W.displaced_icosphere_workload(nu=40, n_queries=n)
    Q = torch.from_numpy(wl.Q).cuda()
    auto = fwn.FastWindingNumber(wl.V, wl.F)
    auto.query(Q)
    none, (w, ins) = _scratch(torch, lambda: auto.query(Q))
    assert none == 0
    if by_config:
        eng, kw = fwn.FastWindingNumber(wl.V, wl.F, traversal=fwn.TRAVERSAL_WARP), {}
    else:
        eng, kw = auto, {"traversal": fwn.TRAVERSAL_WARP}
    some, (w2, ins2) = _scratch(torch, lambda: eng.query(Q, **kw))
    assert some >= 16 * n
    unsorted, (w3, _) = _scratch(torch, lambda: eng.query(Q, sort_queries=0, **kw))
    assert 0 < unsorted < 16 * n
    for a, b in ((w, w2), (w, w3), (ins, ins2)):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
