"""GPU tests of the engines' device memory: destroying an engine beside other work and captures."""
import threading
import time

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


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_destroy_leaves_another_threads_capture_alone(torch, mode):
    """A thread destroys an engine (and builds, queries and destroys another) while this one captures."""
    V, F = W.uv_sphere(16, 8)
    Q = np.random.default_rng(0).uniform(-1.5, 1.5, (5000, 3)).astype(np.float32)
    doomed, kept = fwn.FastWindingNumber(V, F), fwn.FastWindingNumber(V, F)
    want = kept.query(Q)[0]
    x = torch.zeros(8, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    got = []

    def work():
        doomed.close()
        got.append(kept.query(Q)[0])
        another = fwn.FastWindingNumber(V, F)
        got.append(another.query(Q)[0])
        another.close()

    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        x += 1
        t = threading.Thread(target=work)
        t.start()
        t.join()
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    assert len(got) == 2
    for w in got:
        np.testing.assert_array_equal(w, want)


def test_destroy_waits_for_queries_in_flight(torch):
    wl = W.displaced_icosphere_workload(nu=60, n_queries=1_000_000)
    kept, doomed = fwn.FastWindingNumber(wl.V, wl.F), fwn.FastWindingNumber(wl.V, wl.F)
    Q = torch.from_numpy(wl.Q).cuda()
    want = kept.query(Q, traversal=fwn.TRAVERSAL_THREAD)[0]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        got = [doomed.query(Q, traversal=fwn.TRAVERSAL_THREAD)[0] for _ in range(4)]
    doomed.close()
    assert side.query()  # complete
    other = W.displaced_icosphere_workload(nu=61, n_queries=1)
    again = [fwn.FastWindingNumber(other.V, other.F) for _ in range(3)]  # into the same memory
    torch.cuda.synchronize()
    for w in got:
        np.testing.assert_array_equal(w.cpu().numpy(), want.cpu().numpy())
    del again


def test_memory_of_destroyed_engines(torch):
    """Beside more than 2 GiB of live engines a destroyed one's memory stays for the next; of engines
    destroyed together the library keeps 2 GiB at most, without a synchronisation; and that it gives
    back when asked."""
    MB = 1 << 20
    every = fwn.RECORDS_F32 | fwn.RECORDS_F64 | fwn.RECORDS_MOMENTS
    V, F = (torch.from_numpy(x).cuda() for x in W.displaced_icosphere(316, 1))
    make = lambda: fwn.FastWindingNumber(V, F, records=every)  # noqa: E731
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    make().close()
    torch.cuda.synchronize()
    fwn.release_memory()
    nothing = free()
    live = [make() for _ in range(10)]
    size = live[0].info()["device_bytes"]
    assert 10 * size > 4 << 30
    one = make()
    torch.cuda.synchronize()
    beside = free()
    one.close()
    torch.cuda.synchronize()
    assert abs(free() - beside) < 64 * MB
    for e in live:
        e.close()
    temporaries = 1 << 30  # of the builds, kept as well
    assert nothing - free() < (2 << 30) + temporaries
    torch.cuda.synchronize()
    fwn.release_memory()
    assert abs(free() - nothing) < 64 * MB


@pytest.mark.parametrize("mode", ["global", "thread_local"])
@pytest.mark.parametrize("what", ["query", "build"])
def test_thread_ends_beside_a_capture(torch, what, mode):
    """A thread that queried host points, or built an engine, before a capture ends during it: the pinned
    memory that it leaves is freed without breaking the capture."""
    V, F = W.uv_sphere(16, 8)
    eng = fwn.FastWindingNumber(V, F)
    built = []
    ready, go = threading.Event(), threading.Event()

    def work():
        if what == "query":
            eng.query(np.zeros((3, 3), np.float32))
        else:
            built.append(fwn.FastWindingNumber(V, F))
        ready.set()
        go.wait()

    t = threading.Thread(target=work)
    t.start()
    assert ready.wait(60)
    x = torch.zeros(8, device="cuda")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode=mode):
        x += 1
        go.set()
        t.join()
        time.sleep(0.05)  # (the thread's own memory goes after its last Python statement)
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
