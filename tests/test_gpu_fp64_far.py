"""GPU tests of the FP64 form's queries that the whole mesh is far from. Tolerance: that of the FP64
schedules among themselves, 1e-12 in w."""
import math

import numpy as np
import pytest

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

pytestmark = pytest.mark.gpu
FOUR_PI = 4 * math.pi


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return t


def _points(V, n, share):
    """A share of the points far away, the others about the mesh."""
    rng = np.random.default_rng(n)
    Q = W.box_queries(V, n, rng)
    far = rng.random(n) < share
    Q[far] *= 40
    return np.ascontiguousarray(Q, np.float32)


# both sides of the size from which a kernel of their own answers them
@pytest.mark.parametrize("n", [1, 2048, 2049, 30_000])
@pytest.mark.parametrize("share", [0.0, 0.5, 1.0])
def test_matches_thread_schedule(torch, n, share):
    V, F = W.uv_sphere(16, 8)
    eng = fwn.FastWindingNumber(V, F, records=fwn.RECORDS_F64)
    Q = _points(V, n, share)
    Q[:: 7, 0] = [np.nan, np.inf, 3e38][n % 3] if n > 1 else Q[::7, 0]
    Q = torch.from_numpy(Q).cuda()
    w, ins, w64 = eng.query(Q, precision=fwn.PRECISION_FP64, omega_f64=True)
    t, tins, t64 = eng.query(Q, precision=fwn.PRECISION_FP64, omega_f64=True,
                             traversal=fwn.TRAVERSAL_THREAD)
    w64, t64 = w64.cpu().numpy(), t64.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(w64), np.isnan(t64))
    ok = ~np.isnan(t64)
    assert np.max(np.abs(w64 - t64)[ok], initial=0) / FOUR_PI <= 1e-12
    np.testing.assert_array_equal(w.cpu().numpy()[ok], w64[ok].astype(np.float32))
    np.testing.assert_array_equal(ins.cpu().numpy()[ok], (w64[ok].astype(np.float32) > 2 * math.pi))
    alone = torch.cat([eng.query(Q[i:i + 1], precision=fwn.PRECISION_FP64, omega_f64=True)[2]
                       for i in range(min(n, 60))]).cpu().numpy()
    np.testing.assert_array_equal(w64[:60], alone)


def test_not_slower_than_the_thread_schedule(torch):
    """300,000 far queries took 2.8 times the thread schedule's time with a look into the tree each."""
    V, F = W.displaced_icosphere(60, 3)
    eng = fwn.FastWindingNumber(V, F, records=fwn.RECORDS_F64, precision=fwn.PRECISION_FP64)
    Q = torch.from_numpy(_points(V, 300_000, 1.0)).cuda()

    def time(**kw):
        t = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            eng.query(Q, **kw)
            b.record()
            torch.cuda.synchronize()
            t.append(a.elapsed_time(b))
        return sorted(t[2:])[5]

    assert time() <= 1.1 * time(traversal=fwn.TRAVERSAL_THREAD)
