"""The register-tiled z and y passes of planes too large for one block (csrc/dif.cuh) against the
projection in closed form, where their plans change: two and three stages on either axis, odd
lines, partial column tiles and partial line tiles, a single x plane, an axis without a plan
(190 points) beside one with, and the longest y line.  In mixed precision the smaller of these
planes fit one block and the larger take the same passes in float.

Tolerances as for every projection: relative L2 <= 1e-12 in FP64, <= 3e-6 in mixed precision.  Two
solves that differ in their passes alone both meet a residual of 1e-10 (FP64) or 1e-6 of the
stress; their stresses may differ by that times the grains' stiffness contrast (below 4)."""

import numpy as np
import pytest

from materialite_b200.engine import PhaseSpec, SolverHandle, solve
from materialite_b200.microstructure import bunge_random_rotations, periodic_voronoi
from oracle import ssfft_oracle as O
from test_gpu_dif import MASK, reference

pytestmark = pytest.mark.gpu

DIMS = [(2, 256, 256), (3, 175, 189), (1, 225, 250), (2, 243, 147), (2, 190, 175), (2, 175, 190),
        (2, 441, 49), (1, 1000, 35), (7, 245, 180), (4, 135, 125)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 3e-6)])
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_projection(dims, precision, tol):
    tau = np.random.default_rng(sum(dims)).standard_normal((int(np.prod(dims)), 6))
    h = SolverHandle(dims, MASK, precision)
    try:
        out = h.apply_projection(tau).reshape(-1, 6)
    finally:
        h.close()
    ref = reference(dims, tau)
    assert np.linalg.norm(out - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("dims,precision,gtol", [((3, 135, 125), "fp64", 1e-10),
                                                 ((2, 175, 175), "mixed", 1e-6)])
def test_solve_as_on_the_stockham_passes(monkeypatch, dims, precision, gtol):
    rng = np.random.default_rng(5)
    grain = periodic_voronoi(dims, 6, rng).astype(np.int32)
    rotations = bunge_random_rotations(6, rng)
    load = O.LoadOracle.uniaxial(1e-3, "x")
    stress = []
    for off in (None, "1"):
        if off:
            monkeypatch.setenv("SSFFT_NO_PLANE", off)
        h = SolverHandle(dims, load.mask, precision, global_tolerance=gtol,
                         linear_solver_tolerance=0.01 * gtol)
        try:
            h.set_phases([PhaseSpec("elastic", O.cubic_stiffness(250.0, 150.0, 120.0))])
            h.set_microstructure(rotations, grain)
            out, _ = solve(h, load.dstrain, load.dstress, load.stress, end_time=1.0,
                           initial_time_increment=1.0)
            stress.append(np.array(out["stress"]))
        finally:
            h.close()
    assert np.linalg.norm(stress[0] - stress[1]) <= 4 * gtol * np.linalg.norm(stress[1])
