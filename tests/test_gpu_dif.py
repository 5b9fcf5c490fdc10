"""The register-tiled transform passes (csrc/dif.cuh) against the oracle's projection, at the
sizes where their plans change: lines of one radix, two and three stages, odd lines (an extra
column slot), radices with and without a padding slot, partial column tiles of the x pass, the
smallest plane they take and the largest that fits one block in float (160 x 160, 217 KB) and in
double (112 x 112, 218 KB), axes without a plan beside axes with one (11, 13, 17 points), and a
grid of one x plane.

Tolerances as for every projection: relative L2 <= 1e-12 in FP64, <= 3e-6 in mixed precision."""

import numpy as np
import pytest

from oracle import ssfft_oracle as O
from materialite_b200.engine import SolverHandle

pytestmark = pytest.mark.gpu

MASK = np.array([0, 1, 1, 1, 1, 1], dtype=float)
DIMS = [
    (4, 16, 32), (3, 23, 22), (5, 32, 16), (1, 32, 32), (2, 25, 21), (8, 27, 45), (16, 50, 63),
    (9, 35, 49), (7, 81, 20), (30, 28, 27), (45, 8, 75), (48, 36, 40), (64, 16, 36), (75, 18, 30),
    (96, 6, 100), (128, 5, 108), (100, 25, 24), (11, 40, 42), (24, 26, 32), (17, 24, 30),
    (12, 34, 28), (6, 125, 12), (2, 112, 112), (2, 160, 160), (3, 128, 63), (250, 10, 60),
]


def reference(dims, tau):
    """ifftn(Gamma-hat : fftn(tau)).real with Gamma-hat applied in closed form."""
    f = [np.fft.fftfreq(n) for n in dims]
    t = np.stack(np.meshgrid(*(np.tan(np.pi * x) for x in f), indexing="ij"))
    keep = np.ones(dims, dtype=bool)
    for a, n in enumerate(dims):
        if n % 2 == 0:
            np.moveaxis(keep, a, 0)[n // 2] = False
    keep[0, 0, 0] = False
    t = np.where(keep, t, 0.0)
    norm = np.sqrt((t * t).sum(0))
    t = t / np.where(norm > 0, norm, 1.0)
    s = np.fft.fftn(tau.reshape(dims + (6,)), axes=(0, 1, 2))
    mean = s[0, 0, 0] * MASK
    pairs = ((1, 2), (0, 2), (0, 1))
    T = {(i, i): s[..., i] for i in range(3)}
    for k, (i, j) in enumerate(pairs):
        T[i, j] = T[j, i] = s[..., 3 + k] / np.sqrt(2.0)
    u = [sum(T[i, j] * t[j] for j in range(3)) for i in range(3)]
    tu = sum(t[i] * u[i] for i in range(3))
    o = [2 * t[i] * u[i] - tu * t[i] ** 2 for i in range(3)]
    o += [np.sqrt(2.0) * (t[i] * u[j] + u[i] * t[j] - tu * t[i] * t[j]) for i, j in pairs]
    o = np.stack(o, axis=-1)
    o[0, 0, 0] = mean
    return np.fft.ifftn(o, axes=(0, 1, 2)).real.reshape(-1, 6)


def test_reference_is_the_oracle():
    dims = (4, 5, 6)
    tau = np.random.default_rng(1).standard_normal((120, 6))
    ref = O.apply_projection(O.projection_operator(dims, MASK), tau.ravel()).reshape(-1, 6)
    assert np.linalg.norm(reference(dims, tau) - ref) <= 1e-13 * np.linalg.norm(ref)


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
