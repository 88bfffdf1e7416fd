"""GPU tests of the mixed form's near field: the double-float evaluation of ill-conditioned
triangles, the warp walk's list of them and the launch for the groups whose list ran full.

Tolerance: the mixed form's 2e-6 in w against the FP64 form (tests/test_gpu_parity.py), as it holds
for every input there: the near terms are within 2^-30 of the FP64 ones, far below it.
"""
import math

import numpy as np
import pytest

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

pytestmark = pytest.mark.gpu
FOUR_PI = 4 * math.pi
BOTH = fwn.RECORDS_F32 | fwn.RECORDS_F64


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return t


def _pole_queries(n, seed, spread=1e-3):
    """Points around the UV sphere's north pole, where 64 triangles meet: every query is near to
    tens of ill-conditioned triangles."""
    rng = np.random.default_rng(seed)
    return (np.array([0.0, 0.0, 1.0]) + rng.uniform(-spread, spread, (n, 3))).astype(np.float32)


def _w64(eng, torch, Q):
    _, _, w = eng.query(torch.from_numpy(Q).cuda(), precision=fwn.PRECISION_FP64, omega_f64=True)
    return w.cpu().numpy()


# n: one query, both sides of a 32- and a 64-query group, several full lists
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 1000])
@pytest.mark.parametrize("tuning", [1, 3, 5, 6, 7])
def test_pole_cluster(torch, n, tuning):
    V, F = W.uv_sphere(64, 32)
    Q = _pole_queries(n, n)
    eng = fwn.FastWindingNumber(V, F, records=BOTH, tuning=tuning)
    w, _ = eng.query(torch.from_numpy(Q).cuda())
    assert np.max(np.abs(w.cpu().numpy() - _w64(eng, torch, Q))) / FOUR_PI <= 2e-6
    # the answer does not depend on which queries share a group, nor on the schedule variant
    one = fwn.FastWindingNumber(V, F, tuning=3)
    alone = torch.cat([one.query(torch.from_numpy(Q[i:i + 1]).cuda())[0] for i in range(min(n, 40))])
    np.testing.assert_array_equal(w.cpu().numpy()[:40], alone.cpu().numpy())


@pytest.mark.parametrize("tuning", [3, 6])
@pytest.mark.parametrize("cond", [0.0, 4.0])
def test_every_triangle_near(torch, tuning, cond):
    """A near distance beyond the mesh: with cond = 0 every triangle that is not far is evaluated as
    a near one, so every list runs full."""
    wl = W.displaced_icosphere_workload(nu=10, n_queries=3000)
    eng = fwn.FastWindingNumber(wl.V, wl.F, records=BOTH, tuning=tuning, fp64_near_scale=10.0,
                                fp64_cond=cond)
    w, _ = eng.query(torch.from_numpy(wl.Q).cuda())
    assert np.max(np.abs(w.cpu().numpy() - _w64(eng, torch, wl.Q))) / FOUR_PI <= 2e-6


@pytest.mark.parametrize("tuning", [3, 6])
def test_grid_and_forest(torch, tuning):
    """The grid and forest walks leave groups over too, and give the point walk's bits."""
    V, F = W.uv_sphere(64, 32)
    dims, h = (9, 10, 11), 2e-4
    origin = (-4.5 * h, -5 * h, 1 - 5.5 * h)
    eng = fwn.FastWindingNumber(V, F, tuning=tuning)
    wg, _ = eng.query_grid(origin, (h, h, h), dims)
    f32 = np.float32
    ax = [(np.arange(d) + 0.5).astype(np.float64) * float(f32(h)) + float(f32(o))
          for d, o in zip(dims, origin)]
    Z, Y, X = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    Q = np.stack([X.ravel(), Y.ravel(), Z.ravel()], 1).astype(f32)
    wp, _ = eng.query(torch.from_numpy(Q).cuda())
    np.testing.assert_array_equal(wg.reshape(-1).cpu().numpy(), wp.cpu().numpy())
    V2 = np.concatenate([V, V])
    F2 = np.concatenate([F, F])
    forest = fwn.Forest(V2, [0, len(V), 2 * len(V)], F2, [0, len(F), 2 * len(F)], tuning=tuning)
    Qd = torch.from_numpy(np.concatenate([Q[:500], Q])).cuda()
    wf, _ = forest.query_forest(Qd, [0, 500, 500 + len(Q)])
    np.testing.assert_array_equal(wf[500:].cpu().numpy(), wp.cpu().numpy())
    np.testing.assert_array_equal(wf[:500].cpu().numpy(), wp[:500].cpu().numpy())
