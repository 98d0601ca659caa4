"""Aperture deposition at the sizes where its kernel changes form.

The device sums each node's masses in the oracle's order (corner-major, then
quadrature order), so the two agree to the rounding of one fused multiply-add
per term: at most ~1e4 terms of one sign per node, 1.1e-16 each against the
node's own mass, and in practice far less; 1e-13 of the largest mass bounds it.
"""
import numpy as np
import pytest
import torch

from oracle import helmholtz_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,diameter,radial,angular", [
    (1.0e-3, 4.0e-3, 64, 256),   # cell lists, one pass of 16384 points
    (1.0e-3, 3.0e-3, 65, 257),   # 16705 points: a second pass of 321
    (0.2e-3, 9.0e-3, 16, 64),    # 45 nodes across: more cells than the lists hold, key scan
    (0.2e-3, 9.0e-3, 65, 257),   # key scan over two passes
    (1.0e-3, 0.9e-3, 2, 9),      # 18 points: a partial group of four keys
])
def test_deposition_forms(dx, diameter, radial, angular):
    from ultrasound_solver_b200.scene import DeviceOperator, SourceColumns
    n = 60
    full = lambda v: torch.full((n * n * 4,), v, dtype=torch.float64, device="cuda")
    op = DeviceOperator((n, n, 4), dx, 2 * np.pi * 4e4, {"+z": "open"}, full(1.2), full(343.0))
    mid = (n - 1) * dx / 2
    centers = np.array([[mid, mid, 0.0], [mid + 0.37 * dx, mid - 0.81 * dx, 0.0]])
    src = SourceColumns(op, centers, diameter, 1.2, radial, angular)
    got = src.mass_matrix.cpu().numpy()
    want = O.source_mass_matrix((n, n), dx, centers, diameter, radial, angular)
    want = np.asarray(want.todense() if hasattr(want, "todense") else want)
    assert np.abs(got.T - want).max() <= 1e-13 * np.abs(want).max()
    assert np.allclose(got.sum(axis=1), 1.0, rtol=1e-12)
