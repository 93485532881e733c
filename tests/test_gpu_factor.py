"""The one-launch ILU(0) factorisation against the oracle's row-by-row ILU(0)
where its tables can go wrong: one element, one-element-wide boxes, tails of
the 128- and 64-thread column loops, nodes with more than 8 unknowns, many
independent problems and a renumbered mesh.

The matrix has unit diagonals and off-diagonal row sums of at most 1/2
(test_gpu_line_sweeps): no pivot comes near the floor, and an entry's rounding
error is at most twice its update count times eps of the largest entry,
2 * 700 * eps < 2e-13 in FP64 and 1e-4 in FP32 (times 16 unknowns a block)."""
import numpy as np
import pytest

import oracle
from goma_gb300 import problem as pb

from .test_gpu_line_sweeps import cavity, cube, renumbered, system, union

pytestmark = pytest.mark.gpu

CASES = {
    "cavity 1x1": lambda: cavity(1, 1),
    "cavity 1x6": lambda: cavity(1, 6),
    "cavity 13x9": lambda: cavity(13, 9),
    "bratu 6x5": lambda: pb.bratu_square_2d(0, mesh=pb.box_mesh(2, 6, 5)),
    "cube 1x1x1": lambda: cube(1, 1, 1),
    "cube 1x4x1": lambda: cube(1, 4, 1),
    "cube 4x3x3": lambda: cube(4, 3, 3),
    "reacting 3x2x2": lambda: pb.reacting_channel_3d(3, 2, 2),
    "150 cavities 3x2": lambda: union(cavity(3, 2), 150),
    "cube 3x3x2 renumbered by 2": lambda: renumbered(cube(3, 3, 2), 2),
}


@pytest.mark.parametrize("name", list(CASES))
def test_factors_match_the_oracle(name):
    from goma_gb300.newton import GomaNewton
    prob = CASES[name]()
    ija, N, a, _ = system(prob, 5)
    ref = oracle.Oracle(prob).ilu0(a)
    gn = GomaNewton(prob)
    first = None
    for fp32, tol in ((False, 16 * 2e-13), (True, 16 * 1e-4)):
        lu = gn.ilu0_factors(a, fp32=fp32)
        assert np.abs(lu - ref).max() < tol, fp32
        if not fp32:
            first = lu
    # the factors do not depend on timing
    assert np.array_equal(gn.ilu0_factors(a), first)
    gn.close()
