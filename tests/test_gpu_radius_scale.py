"""GPU test of the node radii where squared distances leave float's range."""
import numpy as np
import pytest

import lagrange_gb300 as fwn

pytestmark = pytest.mark.gpu


def test_radius_beyond_floats_squares():
    """A large node's first chunks have vertices whose squared distance from the node's centre is beyond
    float; a chunk that is looked at later has one a little farther, in a group of slots whose own sphere
    is within float. All are slivers without area, centred with the 12 million small triangles, so that
    the facets keep their order and the centre is theirs. The root's radius reaches every vertex."""
    torch = pytest.importorskip("torch")
    n = 12_000_000
    a, b, c = 1.8449e19, 1.8480e19, 4.5e16  # a squared is beyond float, b - c squared is not
    tiny = [[1e15, 0, 0], [-5e14, 1e15, 0], [-5e14, -1e15, 0]]
    V = torch.tensor(tiny + [[a, 0, 0], [-a / 2, 0, 0], [b, 0, 0], [-b / 2 + 1.5 * c, 0, 0],
                             [3 * c, 0, 0], [0, 0, 0], [-2.4e19, -2.4e19, -2.4e19],
                             [2.4e19, 2.4e19, 2.4e19]], device="cuda")
    F = torch.tensor([0, 1, 2], dtype=torch.int32, device="cuda").repeat(n, 1)
    F[:8_000_000:65536] = torch.tensor([3, 4, 4], dtype=torch.int32, device="cuda")
    group = n - 8  # the last group of eight slots: its vertices' mean is near c
    F[group:] = torch.tensor([7, 8, 8], device="cuda")
    F[group] = torch.tensor([5, 6, 6], device="cuda")
    for _ in range(12):  # (which chunk comes first is the GPU's choice)
        eng = fwn.FastWindingNumber(V, F)
        root = eng.export_tree()["center_radius"][0].astype(np.float64)
        far = np.linalg.norm(V[:9].double().cpu().numpy() - root[:3], axis=1).max()
        assert root[3] >= far * (1 - 1e-12)
