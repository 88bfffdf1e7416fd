"""GPU tests of small batches, which take one warp per query: the same bits as the group walk
(tuning 3, which asks for it) over the forms that the rule accepts."""
import ctypes as C

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


def _pair(V, F, **kw):
    """The default engine and one on the same tree that asks for the group walk."""
    return fwn.FastWindingNumber(V, F, **kw), fwn.FastWindingNumber(V, F, tuning=3, **kw)


def _same(torch, a, b, Q):
    Qd = torch.from_numpy(np.ascontiguousarray(Q, np.float32)).cuda()
    (wa, ia), (wb, ib) = a.query(Qd), b.query(Qd)
    np.testing.assert_array_equal(wa.cpu().numpy(), wb.cpu().numpy())
    np.testing.assert_array_equal(ia.cpu().numpy(), ib.cpu().numpy())
    return wa.cpu().numpy(), ia.cpu().numpy()


# leaves of 1 to 16 triangles, every builder, meshes from one triangle up
@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED])
@pytest.mark.parametrize("leaf", [1, 7, 16])
@pytest.mark.parametrize("nu", [1, 12, 60])
def test_matches_group_walk(torch, builder, leaf, nu):
    wl = W.displaced_icosphere_workload(nu=nu, n_queries=1500)
    one, group = _pair(wl.V, wl.F, builder=builder, leaf_size=leaf)
    for n in (1, 2, 5, 1500):
        _same(torch, one, group, wl.Q[:n])


def test_one_triangle(torch):
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], np.float32)
    one, group = _pair(V, np.array([[0, 1, 2]], np.int32))
    Q = np.random.default_rng(0).uniform(-2, 2, (77, 3))
    Q[:3] = V  # on the vertices
    _same(torch, one, group, Q)


# beta: nearly everything far, the default, and every triangle exact (the pending nodes of one
# query then exceed the stack many times over)
@pytest.mark.parametrize("beta", [1e-3, 2.0, 7.0, 1e30])
def test_beta_and_stack(torch, beta):
    wl = W.displaced_icosphere_workload(nu=50, n_queries=200)
    _same(torch, *_pair(wl.V, wl.F, beta=beta, leaf_size=2), wl.Q)


def test_deep_tree_and_odd_points(torch):
    """A spiral whose triangle sizes fall over many decades (a deep, unbalanced tree), and points
    that are not finite."""
    k = np.arange(600)
    r = 0.97 ** k
    P = np.stack([r * np.cos(k), r * np.sin(k), 0.1 * r], 1)
    F = np.stack([k[:-2], k[1:-1], k[2:]], 1)
    Q = np.concatenate([np.random.default_rng(1).uniform(-1, 1, (60, 3)), P[::7]])
    Q[5, 0], Q[6, 1], Q[7, 2] = np.nan, np.inf, -np.inf
    for builder in (fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT):
        _same(torch, *_pair(P, F, leaf_size=1, builder=builder), Q)


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097])
def test_host_buffers(torch, n):
    """Both sides of the staged size, either output alone, and the allocation-free entry."""
    wl = W.displaced_icosphere_workload(nu=20, n_queries=n)
    one, group = _pair(wl.V, wl.F)
    w, ins = _same(torch, one, group, wl.Q)
    hw, hi = one.query(wl.Q)
    np.testing.assert_array_equal(hw, w)
    np.testing.assert_array_equal(hi, ins)
    np.testing.assert_array_equal(one.query(wl.Q, inside=False)[0], w)
    np.testing.assert_array_equal(one.query(wl.Q, omega=False)[1], ins)
    Qd = torch.from_numpy(wl.Q).cuda()
    wn = torch.empty(n, device="cuda")
    fwn._check(fwn.library().fwn_query_noalloc(one.handle, C.c_void_p(Qd.data_ptr()), n,
                                               C.c_void_p(wn.data_ptr()), None, None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(wn.cpu().numpy(), w)


def test_grid_and_forest(torch):
    wl = W.displaced_icosphere_workload(nu=20, n_queries=300)
    one, group = _pair(wl.V, wl.F)
    args = ((-1.2, -1.1, -1.3), (0.17, 0.3, 0.21), (13, 7, 11))
    for a, b in zip(one.query_grid(*args), group.query_grid(*args)):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    V2, F2 = W.uv_sphere(16, 8)
    V, F = np.concatenate([wl.V, V2, wl.V]), np.concatenate([wl.F, F2, wl.F])
    voff = np.cumsum([0, len(wl.V), 0, len(V2), len(wl.V)])   # the second mesh is empty
    foff = np.cumsum([0, len(wl.F), 0, len(F2), len(wl.F)])
    Q = torch.from_numpy(np.concatenate([wl.Q, wl.Q[:50], wl.Q[:77], wl.Q])).cuda()
    qoff = np.cumsum([0, 300, 50, 77, 300])
    res = [fwn.Forest(V, voff, F, foff, tuning=t).query_forest(Q, qoff) for t in (0, 3)]
    for a, b in zip(*res):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    assert not res[0][0][300:350].any()
