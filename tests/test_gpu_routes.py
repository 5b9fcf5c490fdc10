"""Where a grid's route through the transform passes changes (plan.cuh: long_plane, few_planes, the
x pass of single columns and single planes): the projection on both sides of each line against the
closed form, and a request solved alone and in a group, which must agree to the bit.

Tolerances as for every projection: relative L2 <= 1e-12 in FP64, <= 3e-6 in mixed precision."""

import numpy as np
import pytest

from materialite_b200.engine import PhaseSpec, SolverHandle
from materialite_b200.microstructure import bunge_random_rotations
from materialite_b200.serving import RVERequest, RVEServer, run_stream
from oracle import ssfft_oracle as O
from test_gpu_dif import MASK, reference

pytestmark = pytest.mark.gpu

DIMS = [
    # long planes: one round of points (98 | 99 and 49 | 50 x planes), size, ratio, direct sums
    (98, 8, 64), (99, 8, 64), (49, 16, 64), (50, 16, 64), (4, 8, 256), (4, 8, 384), (4, 2, 256),
    (4, 256, 2), (4, 128, 4), (3, 1, 512), (3, 512, 1), (3, 600, 1), (5, 6, 96), (5, 12, 48),
    # few planes of clusters of four (11 | 12), with direct sums, one-block size
    (11, 144, 144), (12, 144, 144), (11, 384, 32), (12, 384, 32), (10, 640, 20), (9, 112, 112),
    (2, 96, 128), (2, 256, 64), (2, 100, 100), (2, 90, 128),
    # a single column on long lines, single planes
    (256, 512, 1), (250, 512, 1), (256, 512, 2), (250, 576, 1), (1, 256, 256), (1, 64, 64), (1, 27, 48),
]


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


@pytest.mark.parametrize("dims", [(6, 8, 64), (2, 128, 128), (4, 128, 256), (1, 32, 32)],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_solve_does_not_depend_on_its_batch(dims, precision):
    """Three requests, the second finished after its first load step, in one group and alone."""
    rng = np.random.default_rng(3)
    V = int(np.prod(dims))

    def requests():
        return [RVERequest(tag=i, dims=dims,
                           phases=[PhaseSpec("elastic", O.cubic_stiffness(250.0, 150.0, 120.0))],
                           rotations=R, grain=g, stress_mask=MASK,
                           strain_rate=np.array([1e-3, 0, 0, 0, 0, 0]), stress_rate=np.zeros(6),
                           dt=1.0, steps=1 if i == 1 else 3, keep_stress=True)
                for i, (R, g) in enumerate(micro)]

    micro = [(bunge_random_rotations(5, rng), rng.integers(0, 5, V).astype(np.int32))
             for _ in range(3)]
    batch = requests()
    srv = RVEServer(max_slots=3, precision=precision)
    comps, _ = run_stream(srv, batch, timeout=120)
    srv.close()
    assert [c.status for c in comps] == [0, 0, 0]
    for one, b in zip(requests(), batch):
        srv = RVEServer(max_slots=1, precision=precision)
        comps, _ = run_stream(srv, [one], timeout=120)
        srv.close()
        assert comps[0].status == 0 and np.array_equal(one.stress, b.stress)
