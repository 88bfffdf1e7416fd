"""GPU tests of the query sort: one launch per pass for few tiles of 2,048 keys, three for more, and
fewer passes for smaller batches. Orders are exact; results do not depend on the order."""
import numpy as np
import pytest

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

pytestmark = pytest.mark.gpu
FEW = 128 * 2048  # the largest batch with one launch per pass


@pytest.fixture(scope="module")
def setup():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    wl = W.displaced_icosphere_workload(nu=16, n_queries=FEW + 5000)
    Q = torch.from_numpy(wl.Q).cuda()
    Q[7] = float("nan")
    Q[1000:4000] = Q[5]  # equal keys keep their order
    return torch, wl, Q


@pytest.mark.parametrize("n", [1, 2, 31, 2047, 2048, 2049, 6000, FEW - 1, FEW])
def test_few_tiles_order(setup, n):
    """A stable sort's order of the first n points is the whole order's, of those points."""
    torch, wl, Q = setup
    eng = fwn.FastWindingNumber(wl.V, wl.F)
    whole = eng.query_order(Q).cpu().numpy().astype(np.int64)
    np.testing.assert_array_equal(np.sort(whole), np.arange(len(Q)))
    part = eng.query_order(Q[:n].contiguous()).cpu().numpy().astype(np.int64)
    np.testing.assert_array_equal(part, whole[whole < n])


@pytest.mark.parametrize("tuning", [1, 6])  # the group walk, at sizes where one warp each is default
@pytest.mark.parametrize("n", [2, 127, 5000, 131_072, 131_073, FEW + 5000])
def test_results_do_not_depend_on_the_sort(setup, n, tuning):
    torch, wl, Q = setup
    eng = fwn.FastWindingNumber(wl.V, wl.F, tuning=tuning)
    q = Q[:n].contiguous()
    w, ins = eng.query(q)[:2]
    w0, ins0 = eng.query(q, sort_queries=0)[:2]
    np.testing.assert_array_equal(w.cpu().numpy(), w0.cpu().numpy())
    assert torch.equal(ins, ins0)


@pytest.mark.parametrize("counts", [(1, 0, 3), (2000, 1, 90_000), (200_000, 0, 150_000)])
def test_forest(setup, counts):
    torch, wl, Q = setup
    V, nv, nf = np.concatenate([wl.V] * 3), len(wl.V), len(wl.F)
    F = np.concatenate([wl.F] * 3)
    voff, foff = np.arange(4) * nv, np.arange(4) * nf
    qoff = np.concatenate([[0], np.cumsum(counts)])
    Qs = torch.cat([Q] * 2)[:qoff[-1]].contiguous()
    one = fwn.FastWindingNumber(wl.V, wl.F, tuning=1).query(Qs)[0].cpu().numpy()
    eng = fwn.Forest(V, voff, F, foff, tuning=1)
    w = eng.query_forest(Qs, qoff)[0].cpu().numpy()
    np.testing.assert_array_equal(w, one)


def test_order_is_the_hilbert_curve(setup):
    """The keys' table against Skilling's algorithm as published (with the exchanges and inversions
    of the lower bits), in Python integers, on cells all over the grid."""
    torch, wl, _ = setup

    def hilbert(X):
        X = list(X)
        q = 512
        while q > 1:
            for i in range(3):
                if X[i] & q:
                    X[0] ^= q - 1
                else:
                    t = (X[0] ^ X[i]) & (q - 1)
                    X[0] ^= t
                    X[i] ^= t
            q >>= 1
        X[1] ^= X[0]
        X[2] ^= X[1]
        t, q = 0, 512
        while q > 1:
            if X[2] & q:
                t ^= q - 1
            q >>= 1
        X = [x ^ t for x in X]
        return sum((X[a] >> b & 1) << (3 * b + 2 - a) for b in range(10) for a in range(3))

    eng = fwn.FastWindingNumber(wl.V, wl.F)
    lo, hi = wl.V.min(0).astype(np.float64), wl.V.max(0).astype(np.float64)
    rng = np.random.default_rng(3)
    cells = rng.integers(0, 1024, size=(20_000, 3))
    # cell centres of the box grown by a quarter of its extent on each side
    Q = lo - 0.25 * (hi - lo) + (cells + 0.5) / 1024 * 1.5 * (hi - lo)
    order = eng.query_order(torch.from_numpy(Q.astype(np.float32)).cuda()).cpu().numpy()
    keys = np.array([hilbert(c) for c in cells.tolist()])
    np.testing.assert_array_equal(order.astype(np.int64), np.argsort(keys, kind="stable"))


@pytest.mark.parametrize("n", [999_999, 1_000_001, 1_000_002])  # omega scattered apart from a million
@pytest.mark.parametrize("shift", [0, 1])                       # aligned outputs and not
def test_scattered_outputs(setup, n, shift):
    torch, wl, Q = setup
    eng = fwn.FastWindingNumber(wl.V, wl.F)
    q = Q.repeat(4, 1)[:n].contiguous()
    w, ins = torch.zeros(n + 1, device="cuda"), torch.zeros(n + 1, dtype=torch.uint8, device="cuda")
    import ctypes as C
    from lagrange_gb300 import _check, _stream_ptr, library
    _check(library().fwn_query(eng.handle, C.c_void_p(q.data_ptr()), n,
                               C.c_void_p(w[shift:].data_ptr()), C.c_void_p(ins[shift:].data_ptr()),
                               _stream_ptr(None)))
    w0, ins0 = eng.query(q, sort_queries=0)[:2]
    np.testing.assert_array_equal(w[shift:shift + n].cpu().numpy(), w0.cpu().numpy())
    assert torch.equal(ins[shift:shift + n], ins0)
