"""Plane passes at the edges of their routes.

* Crystal plasticity (per-point tangents in every Krylov pass) on clusters, asked for and where a
  plane has no register-tiled plan (132 = 11 x 12 points an axis) and no block holds it, and on
  the five register-tiled passes in float (192 x 192: 307 KB in one block).
* The planes that come closest to the 229,376 bytes one block may take: 224 x 125 (229,284) and
  175 x 160 (228,750) in float, 140 x 98 (226,044) in double.
* An elastic solve on register-tiled passes against one on Stockham passes throughout, x included
  (SSFFT_XPASS_THREADS takes the Stockham x pass): both meet a residual of 1e-10 (FP64) or 1e-6
  of the stress, so their stresses may differ by that times the grains' stiffness contrast.
* Three slots of one group in five register-tiled passes, the second with a quarter of the load
  steps, so that its solves are over while its neighbours' go on, against the solver handle.

Tolerances: crystal plasticity FP64 <= 1e-6 and mixed <= 1e-5 of stress and strain against the CPU
oracle, projections 1e-12 and 3e-6, as at the other sizes; slot and handle agree to the bit."""

import numpy as np
import pytest

from materialite_b200.engine import PhaseSpec, SolverHandle
from materialite_b200.serving import RVERequest, RVEServer, run_stream
from test_gpu_dif import MASK, reference
from test_gpu_sizes import C_CUBIC, VOCE, evp_reference, rel_l2, run_evp, schmid, use_cluster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,path,precision,tol", [
    ((4, 128, 128), "cluster8", "fp64", 1e-6), ((4, 128, 128), "cluster8", "mixed", 1e-5),
    ((2, 132, 132), "plane", "fp64", 1e-6), ((2, 132, 132), "plane", "mixed", 1e-5),
    ((2, 192, 192), "plane", "mixed", 1e-5)])
def test_evp(dims, path, precision, tol, monkeypatch):
    use_cluster(monkeypatch, path)
    R, ref = evp_reference(dims, 2)
    out = run_evp(dims, R, 2, precision)
    assert rel_l2(out["stress"], ref["stress"]) < tol
    assert rel_l2(out["strain"], ref["strain"]) < tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 3e-6)])
@pytest.mark.parametrize("dims", [(2, 224, 125), (2, 175, 160), (2, 140, 98)],
                         ids=lambda d: "x".join(map(str, d)))
def test_largest_planes_of_one_block(dims, precision, tol):
    tau = np.random.default_rng(sum(dims)).standard_normal((int(np.prod(dims)), 6))
    h = SolverHandle(dims, MASK, precision)
    try:
        out = h.apply_projection(tau).reshape(-1, 6)
    finally:
        h.close()
    ref = reference(dims, tau)
    assert np.linalg.norm(out - ref) <= tol * np.linalg.norm(ref)


@pytest.mark.parametrize("dims,precision", [((2, 192, 192), "mixed"), ((2, 135, 125), "fp64")])
def test_group_of_five_pass_solves(dims, precision):
    from materialite_b200.microstructure import bunge_random_rotations
    rng = np.random.default_rng(8)
    V = int(np.prod(dims))
    phase = PhaseSpec("evp", C_CUBIC, schmid(), 1e-3, 20.0, 0.1, "voce", VOCE, 1.0)
    rate = np.array([1e-3, 0, 0, 0, 0, 0])
    reqs = [RVERequest(tag=i, dims=dims, phases=[phase], rotations=bunge_random_rotations(6, rng),
                       grain=rng.integers(0, 6, V).astype(np.int32), stress_mask=MASK,
                       strain_rate=rate, stress_rate=np.zeros(6), dt=0.25,
                       steps=1 if i == 1 else 4, keep_stress=True) for i in range(3)]
    srv = RVEServer(max_slots=3, precision=precision, krylov_floor=0.0, krylov_forcing=0.0)
    comps, _ = run_stream(srv, reqs, timeout=300)
    srv.close()
    assert [c.status for c in comps] == [0, 0, 0]
    for r in reqs:
        h = SolverHandle(dims, MASK, precision, global_tolerance=r.global_tolerance,
                         linear_solver_tolerance=r.linear_solver_tolerance)
        try:
            h.set_phases(r.phases)
            h.set_microstructure(r.rotations, r.grain)
            h.solve_constant_rates(r.strain_rate, r.stress_rate, r.dt * r.steps, r.dt)
            assert np.array_equal(h.field("stress"), r.stress)
        finally:
            h.close()


@pytest.mark.parametrize("dims,precision,gtol", [((3, 135, 125), "fp64", 1e-10),
                                                 ((24, 20, 27), "fp64", 1e-10),
                                                 ((2, 192, 175), "mixed", 1e-6),
                                                 ((20, 45, 40), "mixed", 1e-6)])
def test_solve_as_on_stockham_passes_throughout(monkeypatch, dims, precision, gtol):
    from materialite_b200.microstructure import bunge_random_rotations, periodic_voronoi
    rng = np.random.default_rng(5)
    grain = periodic_voronoi(dims, 6, rng).astype(np.int32)
    rotations = bunge_random_rotations(6, rng)
    stress = []
    for stockham in (False, True):
        if stockham:
            monkeypatch.setenv("SSFFT_NO_PLANE", "1")
            monkeypatch.setenv("SSFFT_XPASS_THREADS", "192")
        h = SolverHandle(dims, MASK, precision, global_tolerance=gtol,
                         linear_solver_tolerance=0.01 * gtol)
        try:
            h.set_phases([PhaseSpec("elastic", C_CUBIC)])
            h.set_microstructure(rotations, grain)
            h.solve_constant_rates(np.array([1e-3, 0, 0, 0, 0, 0]), np.zeros(6), 1.0, 1.0)
            stress.append(h.field("stress"))
        finally:
            h.close()
    assert np.linalg.norm(stress[0] - stress[1]) <= 4 * gtol * np.linalg.norm(stress[1])
