"""GPU test of the FP64 form's complex products (default schedule): they stay in range whatever
triangles contribute nothing to them. Tolerance: that of the FP64 schedules among themselves, 1e-12 in
w per unit of the sum (the sum here is of 40,000 equal angles)."""
import math

import numpy as np
import pytest

import lagrange_gb300 as fwn

pytestmark = pytest.mark.gpu


def test_many_triangles_with_flat_ones_at_the_rescaling():
    """A query's triangles go to 32 products in turn, whose factors here are 2^0.98 each; the triangles
    of every 256th round lie in the plane of the query. (All centroids are equal, so the tree keeps
    the facets' order.)"""
    torch = pytest.importorskip("torch")
    n = 40_000
    V = np.array([[20, 0, 0], [20, 3, 0], [20, 0, 3], [20, 1, 1], [20, 2, 2]], np.float32)
    F = np.tile(np.array([[0, 1, 2]], np.int32), (n, 1))
    flat = (np.arange(n) // 32) % 256 == 255
    F[flat] = [0, 3, 4]
    eng = fwn.FastWindingNumber(V, F, records=fwn.RECORDS_F64, beta=1e30)
    Q = torch.zeros((3, 3), device="cuda")
    _, _, w = eng.query(Q, precision=fwn.PRECISION_FP64, omega_f64=True)
    a, b, c = (v.astype(np.float64) for v in V[:3])
    la, lb, lc = (np.linalg.norm(x) for x in (a, b, c))
    one = 2 * math.atan2(a @ np.cross(b, c), la * lb * lc + a @ b * lc + b @ c * la + c @ a * lb)
    want = (n - int(flat.sum())) * one
    assert np.max(np.abs(w.cpu().numpy() - want)) <= 1e-12 * abs(want)
