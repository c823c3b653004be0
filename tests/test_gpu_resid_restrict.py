"""The colour-0 residual and its restriction in one kernel
(k_resid_restrict0) write the separate kernels' bits on every level."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# odd and even extents in each axis, axes of two and three nodes, rows of one
# group and of three rows a block (1352) and past that (1400: the separate
# kernels), one tile of coarse rows and several, one problem and many
@pytest.mark.parametrize("shape,n", [((34, 33, 35), 1), ((65, 66, 64), 3), ((40, 3, 300), 2),
                                     ((2, 40, 90), 2), ((90, 41, 2), 3), ((9, 10, 1352), 2),
                                     ((9, 10, 1400), 1), ((48, 200, 16), 12)])
def test_one_pass_gives_the_separate_kernels_bits(shape, n):
    from ion_gym_gb300 import _lib
    from ion_gym_gb300.physics.mixed import MixedSession
    rng = np.random.default_rng(4)
    masks = []
    for _ in range(n):
        m = rng.random(shape) < 0.03
        masks.append(m)
    metal = np.any(masks, 0)
    with MixedSession(metal, n) as s:
        s.solve_bases(masks, 1.0, 1e-6)
        bad = (ctypes.c_longlong * 8)(*([-1] * 8))
        _lib.check(_lib.lib().ig_mixed_check_fused(s._h, n, bad), "ig_mixed_check_fused")
    assert list(bad) == [0] * 8
