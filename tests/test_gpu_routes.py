"""GPU tests of which walk a batch takes."""
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


def _batches(V, F, n, seed=1):
    """n points in the box, half of them near the surface, all near it, in a slice, about a vertex."""
    rng = np.random.default_rng(seed)
    box = W.box_queries(V, n, rng)
    near = W.surface_queries(V, F, n, rng, 1e-6, 1e-3)
    flat = box * np.float32([1, 1, 0])
    part = V[len(V) // 3] + rng.uniform(-1e-3, 1e-3, (n, 3))
    mixed = np.where(rng.random(n)[:, None] < 0.5, near, box)
    return {k: np.ascontiguousarray(q, np.float32) for k, q in
            {"box": box, "mixed": mixed, "near": near, "slice": flat, "vertex": part}.items()}


def _time(torch, f):
    t = []
    for _ in range(12):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        t.append(a.elapsed_time(b))
    return sorted(t[2:])[5]


def test_batches_that_lie_together_are_not_slower_than_groups(torch):
    """A slice of a large mesh and the surroundings of a vertex: one warp per query took 2.1 and 2.8 times
    the group walk's time."""
    V, F = W.displaced_icosphere(316, 3)
    auto, group = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F, tuning=3)
    for name, Q in _batches(V, F, 150_000).items():
        Q = torch.from_numpy(Q).cuda()
        assert _time(torch, lambda: auto.query(Q)) <= 1.5 * _time(torch, lambda: group.query(Q)), name


# around the sure line and the limit (75,000 on this tree) of the rule, every kind of batch
@pytest.mark.parametrize("n", [30_000, 30_001, 45_000, 74_000, 80_000])
def test_same_bits_around_the_lines(torch, n):
    V, F = W.displaced_icosphere(100, 3)
    auto, group = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F, tuning=3)
    for Q in _batches(V, F, n).values():
        Qd = torch.from_numpy(Q).cuda()
        w, ins = (x.cpu().numpy() for x in group.query(Qd))
        for got in (auto.query(Qd), auto.query(Qd, sort_queries=0), auto.query(Qd, inside=False),
                    auto.query(Q), auto.query(Qd, omega=False)):
            for x, want in zip(got, (w, ins)):
                if x is not None:
                    np.testing.assert_array_equal(x if isinstance(x, np.ndarray) else x.cpu().numpy(), want)
        wn, ni = torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.uint8, device="cuda")
        fwn._check(fwn.library().fwn_query_noalloc(auto.handle, *(C.c_void_p(x) for x in (
            Qd.data_ptr(),)), n, C.c_void_p(wn.data_ptr()), C.c_void_p(ni.data_ptr()), None))
        torch.cuda.synchronize()
        np.testing.assert_array_equal(wn.cpu().numpy(), w)
        np.testing.assert_array_equal(ni.cpu().numpy(), ins)


def test_choice_is_made_at_each_replay(torch):
    """A captured query decides for the points that it finds, not for those of the capture."""
    n = 60_000
    V, F = W.displaced_icosphere(100, 3)
    auto, group = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F, tuning=3)
    batches = _batches(V, F, n)
    Q = torch.from_numpy(batches["box"]).cuda()
    w = torch.empty(n, device="cuda")
    L, stream = fwn.library(), torch.cuda.Stream()
    call = lambda: fwn._check(L.fwn_query(auto.handle, C.c_void_p(Q.data_ptr()), n,  # noqa: E731
                                          C.c_void_p(w.data_ptr()), None, C.c_void_p(stream.cuda_stream)))
    torch.cuda.synchronize()
    call()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    for name in ("vertex", "mixed", "slice", "box"):
        Q.copy_(torch.from_numpy(batches[name]))
        w.fill_(7.0)
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(w.cpu().numpy(), group.query(Q)[0].cpu().numpy())


@pytest.mark.parametrize("half", [1.2, 0.01])
@pytest.mark.parametrize("dims", [(34, 35, 36), (36, 40, 31)])
def test_grids_around_the_lines(torch, half, dims):
    V, F = W.displaced_icosphere(100, 3)
    auto, group = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F, tuning=3)
    h = [2 * half / d for d in dims]
    for a, b in zip(auto.query_grid((-half, -half, 1 - half), h, dims),
                    group.query_grid((-half, -half, 1 - half), h, dims)):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())


@pytest.mark.parametrize("meshes", [2, 70])  # narrow sort keys, and wide ones
@pytest.mark.parametrize("kind", ["box", "vertex"])
def test_forests_around_the_lines(torch, meshes, kind):
    V, F = W.displaced_icosphere(40, 3)
    m = np.arange(meshes)
    Vs, Fs = np.tile(V, (meshes, 1)), np.tile(F, (meshes, 1))
    each = 36_000 // meshes
    Q = torch.from_numpy(np.tile(_batches(V, F, each)[kind], (meshes, 1))).cuda()
    off = lambda k: np.append(m, meshes) * k  # noqa: E731
    res = [fwn.Forest(Vs, off(len(V)), Fs, off(len(F)), tuning=t).query_forest(Q, off(each)) for t in (0, 3)]
    for a, b in zip(*res):
        np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())


@pytest.mark.parametrize("n,kw", [
    (20_000, {"precision": fwn.PRECISION_FP64, "traversal": fwn.TRAVERSAL_WARP}),
    (20_000, {"precision": fwn.PRECISION_FP64, "traversal": fwn.TRAVERSAL_THREAD}),
    (100_000, {"beta": 3.0, "traversal": fwn.TRAVERSAL_WARP})])
def test_sorted_walks_are_as_fast_as_ordered_ones(torch, n, kw):
    """A walk after the sort takes the time of a walk over points that are in that order already, and the
    sort's (60 us at most). Launches that overlapped the sort's end made the FP64 ones 1.17 and 1.22 times as long."""
    V, F = W.displaced_icosphere(158, 3)
    eng = fwn.FastWindingNumber(V, F, records=fwn.RECORDS_F32 | fwn.RECORDS_F64)
    Q = torch.from_numpy(_batches(V, F, n)["mixed"]).cuda()
    ordered = Q[eng.query_order(Q).long()].contiguous()
    walk = _time(torch, lambda: eng.query(ordered, sort_queries=0, **kw))
    assert _time(torch, lambda: eng.query(Q, **kw)) <= 1.1 * walk + 0.06


def test_far_batches_take_a_warp_each(torch):
    """Points outside the mesh's frame fall into its outer cells, but their walks are short: 45,000 took 67
    us with a warp each and 146 in groups."""
    n = 45_000
    V, F = W.displaced_icosphere(158, 3)
    auto, group = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F, tuning=3)
    Q = torch.from_numpy(_batches(V, F, n)["box"] * np.float32(40)).cuda()
    np.testing.assert_array_equal(auto.query(Q)[0].cpu().numpy(), group.query(Q)[0].cpu().numpy())
    assert _time(torch, lambda: auto.query(Q)) <= 0.9 * _time(torch, lambda: group.query(Q))


@pytest.mark.parametrize("n", [33, 100_000])
def test_counting_costs_little(torch, n):
    """The walk with counters, one query per lane: it took 1.3 to 1.45 times the plain walk's time."""
    V, F = W.displaced_icosphere(158, 3)
    eng = fwn.FastWindingNumber(V, F, tuning=3)
    Q = torch.from_numpy(_batches(V, F, n)["mixed"]).cuda()
    plain = _time(torch, lambda: eng.query(Q))
    assert _time(torch, lambda: eng.query(Q, stats=True)) <= 1.12 * plain + 0.06
