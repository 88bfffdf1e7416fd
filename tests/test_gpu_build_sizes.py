"""GPU tests of the build at sizes where its kernels change form: levels of a few nodes and of
thousands (the refit's lane and thread forms), triangles without area, and meshes around the
split builders' whole-block segments. Against the CPU restatement of the build: topology, order,
centres and radii bit for bit; FP64 moments to 1e-12 of their largest (tests/test_gpu_parity.py)."""
import numpy as np
import pytest

import lagrange_gb300 as fwn
from lagrange_gb300 import workloads as W

pytestmark = pytest.mark.gpu
ALL = fwn.RECORDS_F32 | fwn.RECORDS_F64 | fwn.RECORDS_MOMENTS


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("needs a CUDA device")
    return t


def _compare(oracle_mod, V, F, leaf, builder):
    got = fwn.FastWindingNumber(V, F, records=ALL, leaf_size=leaf, builder=builder)
    m, got = got.export_moments(), got.export_tree()
    ref = oracle_mod.LbvhTree(V, F, leaf_size=leaf, builder=builder).export()
    for k in ("skip", "tri_begin", "tri_count", "sorted_tri", "mesh_root"):
        np.testing.assert_array_equal(got[k], ref[k], err_msg=k)
    np.testing.assert_array_equal(got["center_radius"], ref["center_radius"])
    scale = np.max(np.abs(ref["moments"]), axis=0) + 1e-300
    assert np.max(np.abs(m - ref["moments"]) / scale) <= 1e-12


@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED])
@pytest.mark.parametrize("n", [1, 2, 3, 9, 17, 33, 257, 1024, 1025, 2049, 5000])
def test_small_levels(torch, oracle_mod, builder, n):
    """n random triangles, a third of them without area (the centre falls back to plain means)."""
    rng = np.random.default_rng(n)
    V = rng.normal(size=(3 * n, 3)).astype(np.float32)
    V[1::9] = V[0::9][:len(V[1::9])]
    V[2::9] = V[0::9][:len(V[2::9])]
    _compare(oracle_mod, V, np.arange(3 * n, dtype=np.int32).reshape(-1, 3), 1, builder)


@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED])
def test_large_levels(torch, oracle_mod, builder):
    """51,200 triangles, one per leaf: levels on both sides of the refit's change of form."""
    wl = W.displaced_icosphere_workload(nu=50, n_queries=1)
    assert len(wl.F) > 4 * 8192
    _compare(oracle_mod, wl.V, wl.F, 1, builder)


@pytest.mark.parametrize("builder", [fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED])
@pytest.mark.parametrize("n", [1500, 6000])
def test_coincident_centroids(torch, oracle_mod, builder, n):
    """Every centroid in one place (splits by position), and one far away (splits of one)."""
    rng = np.random.default_rng(7)
    T = rng.integers(-4, 5, size=(n, 3, 3)).astype(np.float32)
    T[:, 2] = -T[:, 0] - T[:, 1]  # centroids at the origin, exactly
    T[0] += 1000
    _compare(oracle_mod, T.reshape(-1, 3), np.arange(3 * n, dtype=np.int32).reshape(-1, 3), 4, builder)


def test_engine_memory_is_reused_safely(torch):
    """An engine destroyed while a query on another stream still reads it: the query is right, and
    so are the engines that take over its memory; builds from several threads, too."""
    import threading
    wl = W.displaced_icosphere_workload(nu=60, n_queries=400_000)
    Q = torch.from_numpy(wl.Q).cuda()
    w0 = fwn.FastWindingNumber(wl.V, wl.F).query(Q)[0].clone()
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(3):
        eng = fwn.FastWindingNumber(wl.V, wl.F)
        with torch.cuda.stream(side):
            w = eng.query(Q)[0]
        eng.close()
        other = fwn.FastWindingNumber(wl.V * 2, wl.F)  # other values in the same memory
        side.synchronize()
        assert torch.equal(w, w0)
        del other
    out = [None] * 4

    def work(i):
        for _ in range(3):
            out[i] = fwn.FastWindingNumber(wl.V, wl.F, builder=i % 3).info()["num_nodes"]
    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert out[0] == out[3] and all(out)


def test_build_in_capture_is_refused(torch):
    wl = W.uv_sphere_workload(n_queries=1)
    V, F = torch.from_numpy(wl.V).cuda(), torch.from_numpy(wl.F.astype(np.int32)).cuda()
    x = torch.zeros(4, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        x += 1
        with pytest.raises(fwn.WindingError):
            fwn.FastWindingNumber(V, F)
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1, 1, 1, 1]


@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT])
@pytest.mark.parametrize("scale,shift", [(1e-20, 0), (1e-12, 0), (1e17, 0), (1.0, 3e4), (1e-3, 30.0)])
def test_radii_at_scales(torch, oracle_mod, builder, scale, shift):
    """Squared lengths at both ends of float (every vertex is looked at there), and meshes far from
    the origin, where the group spheres' centres round coarsely; a sphere (every vertex of the root
    is a candidate) with some long triangles."""
    wl = W.displaced_icosphere_workload(nu=20, n_queries=1)
    V, F = wl.V.astype(np.float64), wl.F.copy()
    F[::97, 1] = F[0, 0]
    _compare(oracle_mod, ((V + shift) * scale).astype(np.float32), F, 4, builder)


@pytest.mark.parametrize("builder", [fwn.BUILDER_LBVH, fwn.BUILDER_SPLIT, fwn.BUILDER_BINNED])
@pytest.mark.parametrize("fault", ["nan", "inf", "index", "negative"])
def test_bad_input_of_a_large_mesh(torch, builder, fault):
    """The levels that are launched before the input's check has come back run on whatever the bad
    triangles gave; the build is refused, and the next one is right."""
    wl = W.displaced_icosphere_workload(nu=60, n_queries=1)
    V, F = wl.V.copy(), wl.F.copy()
    if fault == "nan":
        V[F[5000, 1]] = np.nan
    elif fault == "inf":
        V[F[123, 0]] = (np.inf, 0, -np.inf)
    else:
        F[7777, 2] = len(V) if fault == "index" else -1
    good = fwn.FastWindingNumber(wl.V, wl.F, builder=builder).export_tree()
    with pytest.raises(fwn.WindingError):
        fwn.FastWindingNumber(V, F, builder=builder)
    again = fwn.FastWindingNumber(wl.V, wl.F, builder=builder).export_tree()
    for k in good:
        np.testing.assert_array_equal(good[k], again[k])
