"""The byte model of bench.py counts the y passes that a float Krylov iteration really has."""

import numpy as np
import pytest

import bench
from materialite_b200.engine import PhaseSpec, SolverHandle


def test_y_passes_of_cubes():
    # one block up to 160^3, five passes from 162^3; 130 = 2 5 13 and 132 = 12 11 on clusters
    sizes = (16, 64, 128, 130, 132, 160, 162, 168, 175, 192, 256, 512)
    assert [bench.separate_y_passes(n) for n in sizes] == [False] * 6 + [True] * 6


@pytest.mark.parametrize("n,columns", [(192, 96), (256, 128), (175, 88)])
def test_byte_model_of_five_passes(n, columns):
    b = bench.kernel_bytes_per_voxel(n)
    assert b["yfwd"] == b["yinv"] == pytest.approx(2 * 6 * columns / n * 8.0)
    assert bench.kernel_bytes_per_voxel(n, y_passes=False)["yfwd"] == 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 64, 128, 132, 160, 162, 168, 192])
def test_rule_is_the_library_s(n):
    """A Krylov iteration is the update, the epilogue and three or five transform kernels."""
    h = SolverHandle((n, n, n), np.array([0, 1, 1, 1, 1, 1.0]), "mixed", global_tolerance=1e-6,
                     linear_solver_tolerance=1e-8)
    try:
        h.set_phases([PhaseSpec("elastic", bench.cubic_mandel(250.0, 150.0, 120.0))])
        grain = np.random.default_rng(1).integers(0, 4, n ** 3).astype(np.int32)
        q = np.linalg.qr(np.random.default_rng(2).standard_normal((4, 3, 3)))[0]
        h.set_microstructure(q * np.sign(np.linalg.det(q))[:, None, None], grain)
        h.solve_constant_rates(np.array([1e-3, 0, 0, 0, 0, 0]), np.zeros(6), 1.0, 1.0)
        assert bench.kernels_per_iteration(h) == (7 if bench.separate_y_passes(n) else 5)
    finally:
        h.close()
