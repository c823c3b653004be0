"""The cluster launch of the small levels and the step of three directions do
run where the tests that compare them with the separate launches mean them
to: counted by the launches, and by the bytes a step is said to move."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _session(env, metal, n):
    from ion_gym_gb300.physics.mixed import MixedSession
    os.environ.update(env)
    try:
        return MixedSession(metal, n)
    finally:
        for k in env:
            del os.environ[k]


def _deck(shape, n):
    masks = []
    for q in range(n):
        m = np.zeros(shape, bool)
        m[4 + 5 * q:7 + 5 * q, 3:9, 5:20] = True
        masks.append(m)
    return masks, np.any(masks, 0)


@pytest.mark.parametrize("n_b,levels", [(3, 2), (24, 1)])
def test_the_cluster_takes_the_small_levels(n_b, levels):
    """60^3 has two levels between the finest and the bottom; with cycles of
    2 + 2 pairs each takes 9 launches a cycle (3 and 4 half-sweeps, residual
    with restriction, prolongation), the bottom one.  The clusters of three
    problems take both levels; those of 24 are not resident at once (8 CTAs
    each on 152 SMs), so that only the last level and the bottom are one launch
    (k_tail_cycle)."""
    from ion_gym_gb300 import _lib
    masks, metal = _deck((60, 60, 60), 3)
    masks = (masks * 8)[:n_b]
    n, steps = {}, {}
    for tail in ("0", "1"):
        with _session({"IG_MIXED_TAIL": tail, "IG_MIXED_TB_LEVELS": "0"}, metal, n_b) as s:
            s.set_cycle(2, 2, 3)
            s.solve_bases(masks, 1.0, 1e-9)
            before = _lib.lib().ig_mixed_launch_count()
            s.solve_bases(masks, 1.0, 1e-9)
            n[tail] = _lib.lib().ig_mixed_launch_count() - before
            steps[tail] = s.last_steps
    assert steps["0"] == steps["1"] > 0
    visits = 2 if n_b >= 4 else 1  # of the first coarse level (the batches' default)
    assert n["0"] - n["1"] == steps["1"] * 3 * visits * levels * 9


@pytest.mark.parametrize("shape,n_b", [((12, 20, 210), 1), ((18, 33, 197), 5), ((40, 31, 33), 2)])
def test_three_directions(shape, n_b):
    """Folding alone saves 16 bytes a node and step, keeping the directions
    another 8."""
    rng = np.random.default_rng(shape[0])
    metal = rng.random(shape) < 0.02
    b = {}
    for fold in ("0", "1"):
        with _session({"IG_MIXED_FOLD": fold, "IG_MIXED_TB_LEVELS": "0"}, metal, n_b) as s:
            s.set_cycle(2, 2, 3)
            b[fold] = s.step_bytes(1)
    assert b["0"] - b["1"] == 24.0 * np.prod(shape)
