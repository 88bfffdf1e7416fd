"""GPU tests of the FP64 form's default schedule (one warp per query, angles summed as complex
numbers) against the plain thread schedule, which sums the same terms one by one. Tolerance: 1e-12
in w, that of the FP64 schedules among themselves (tests/test_gpu_parity.py)."""
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


def _compare(torch, eng, Q):
    Qd = torch.from_numpy(np.ascontiguousarray(Q, np.float32)).cuda()
    w, ins, w64 = eng.query(Qd, precision=fwn.PRECISION_FP64, omega_f64=True)
    _, ins_t, t64 = eng.query(Qd, precision=fwn.PRECISION_FP64, omega_f64=True,
                              traversal=fwn.TRAVERSAL_THREAD)
    w64, t64 = w64.cpu().numpy(), t64.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(w64), np.isnan(t64))
    ok = ~np.isnan(t64)
    assert np.max(np.abs(w64 - t64)[ok], initial=0) / FOUR_PI <= 1e-12
    np.testing.assert_array_equal(w.cpu().numpy()[ok], w64[ok].astype(np.float32))
    sure = ok & (np.abs(t64 / FOUR_PI - 0.5) > 1e-6)
    np.testing.assert_array_equal(ins.cpu().numpy()[sure], ins_t.cpu().numpy()[sure])
    # a query's answer does not depend on its batch
    k = min(len(Q), 40)
    alone = torch.cat([eng.query(Qd[i:i + 1], precision=fwn.PRECISION_FP64, omega_f64=True)[2]
                       for i in range(k)]).cpu().numpy()
    np.testing.assert_array_equal(w64[:k], alone)


@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT])
@pytest.mark.parametrize("leaf", [1, 7, 16])
@pytest.mark.parametrize("n", [1, 33, 2000, 25_000])  # 25,000: runs of more than one query
def test_matches_thread_schedule(torch, builder, leaf, n):
    wl = W.displaced_icosphere_workload(nu=30, n_queries=n)
    _compare(torch, fwn.FastWindingNumber(wl.V, wl.F, records=fwn.RECORDS_F64, builder=builder,
                                          leaf_size=leaf), wl.Q)


# every triangle exact (many whole turns of the product), and a soup with flipped facets
@pytest.mark.parametrize("beta", [0.5, 2.0, 1e30])
def test_beta_and_soup(torch, beta):
    wl = W.defective_soup_workload(nu=12, n_queries=1500)
    _compare(torch, fwn.FastWindingNumber(wl.V, wl.F, records=fwn.RECORDS_F64, beta=beta), wl.Q)


# scales at both ends of the squared lengths that the Newton steps take, and beyond them
@pytest.mark.parametrize("scale", [1e-18, 1e-10, 1.0, 1e12])
def test_special_points(torch, scale):
    """Vertices, edge and facet midpoints (in their triangles' planes), far points and points that
    are not finite."""
    V, F = W.uv_sphere(16, 8)
    mid = V[F].mean(1)
    edge = (V[F[:, 0]] + V[F[:, 1]]) / 2
    Q = np.concatenate([V, mid, edge, 50 * V[:9], np.zeros((1, 3))]) * scale
    bad = np.array([[np.nan, 0, 0], [np.inf, 0, 0], [0, -np.inf, 1]])
    eng = fwn.FastWindingNumber(V * scale, F, records=fwn.RECORDS_F64, beta=1e30)
    _compare(torch, eng, np.concatenate([Q, bad]))


# queries of a few terms and of many, next to each other: batches that hold several queries' terms
@pytest.mark.parametrize("n", [5, 4 * 152 * 128 + 3, 200_000])
def test_mixed_neighbours(torch, n):
    wl = W.displaced_icosphere_workload(nu=20, n_queries=n)
    Q = wl.Q.copy()
    Q[::3] = Q[::3] * 40 + 200  # far away: the root's term alone
    Q[1::7] = wl.V[np.arange(len(Q[1::7])) % len(wl.V)]  # on vertices
    _compare(torch, fwn.FastWindingNumber(wl.V, wl.F, records=fwn.RECORDS_F64, leaf_size=16), Q)
