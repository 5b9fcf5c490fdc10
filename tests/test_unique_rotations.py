"""Distinct rotations of a microstructure (engine.unique_rotations)."""

import numpy as np
import pytest


@pytest.mark.parametrize("points,grains", [(0, 1), (1, 1), (7, 3), (3000, 2), (3000, 40), (500, 500)])
def test_unique_rotations_are_numpys(points, grains):
    """The distinct rotations and the index of each point, as np.unique over the rows gives
    them, where rows repeat (the hashed path) and where they do not, with signed zeros."""
    from materialite_b200.engine import unique_rotations
    from materialite_b200.microstructure import quaternion_random_rotations
    rng = np.random.default_rng(points + grains)
    pool = quaternion_random_rotations(grains, rng)
    R = pool[rng.integers(0, grains, points)] if grains < max(points, 1) else pool[:points]
    if points > 6:
        R[2] = np.eye(3)
        R[5] = np.where(np.eye(3) > 0, 1.0, -0.0)
    table, index = unique_rotations(R)
    want, inverse = np.unique(R.reshape(-1, 9), axis=0, return_inverse=True)
    assert np.array_equal(table, want.reshape(-1, 3, 3))
    assert np.array_equal(index, inverse.reshape(-1)) and index.dtype == np.int32
