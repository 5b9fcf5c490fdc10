"""Sums over many slots of a launch: a block takes several chunks of a slot in a row where a group
has many (krylov.cuh: chunk_groups), and results stay those of the slot alone, bit for bit.  Sizes
with chunks of 256, 512, 768, 1024 and 4096 points, of a last chunk that is partial, and (33 x 31 x
35, an odd number of points) without 16-byte loads; 5 and 16 slots; strain and stress rates."""

import numpy as np
import pytest

from materialite_b200.engine import PhaseSpec, SolverHandle
from materialite_b200.microstructure import bunge_random_rotations
from materialite_b200.serving import RVERequest, RVEServer, run_stream
from test_gpu_dif import MASK
from test_gpu_sizes import C_CUBIC, VOCE, schmid

pytestmark = pytest.mark.gpu

ELASTIC = PhaseSpec("elastic", C_CUBIC)
EVP = PhaseSpec("evp", C_CUBIC, schmid(), 1e-3, 20.0, 0.1, "voce", VOCE, 1.0)


@pytest.mark.parametrize("dims,precision,phase,slots", [
    ((32, 32, 32), "mixed", EVP, 16), ((32, 32, 32), "fp64", ELASTIC, 16),
    ((33, 31, 35), "mixed", EVP, 16), ((33, 31, 35), "fp64", EVP, 5),
    ((40, 50, 50), "mixed", ELASTIC, 16), ((60, 60, 55), "mixed", EVP, 5),
    ((64, 64, 64), "mixed", ELASTIC, 16), ((72, 72, 60), "fp64", ELASTIC, 5),
    ((135, 140, 128), "mixed", ELASTIC, 5)], ids=str)
def test_a_slot_is_as_alone(dims, precision, phase, slots):
    rng = np.random.default_rng(12)
    V = int(np.prod(dims))
    rate, stress_rate = np.array([1e-3, 0, 0, 0, 0, 0]), np.array([0, 2e-3, 0, 0, 0, 0])
    reqs = [RVERequest(tag=i, dims=dims, phases=[phase], rotations=bunge_random_rotations(6, rng),
                       grain=rng.integers(0, 6, V).astype(np.int32), stress_mask=MASK,
                       strain_rate=rate, stress_rate=stress_rate, dt=0.25,
                       steps=1 + i % 3, keep_stress=True) for i in range(slots)]
    srv = RVEServer(max_slots=slots, precision=precision, krylov_floor=0.0, krylov_forcing=0.0)
    comps, _ = run_stream(srv, reqs, timeout=300)
    srv.close()
    assert all(c.status == 0 for c in comps)
    for r in reqs[::4]:
        h = SolverHandle(dims, MASK, precision, global_tolerance=r.global_tolerance,
                         linear_solver_tolerance=r.linear_solver_tolerance)
        try:
            h.set_phases(r.phases)
            h.set_microstructure(r.rotations, r.grain)
            h.solve_constant_rates(r.strain_rate, r.stress_rate, r.dt * r.steps, r.dt)
            assert np.array_equal(h.field("stress"), r.stress)
        finally:
            h.close()
