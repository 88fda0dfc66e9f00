"""The smallest point levels in one launch (kernels_small.cu) and the first
smoothing step taken by the producer of a level's rhs, against the C
restatement of the reference, which they must equal bit for bit: finest levels
just below and above the launch's size limit (the whole cycle in it, or the
levels below), more and less than 32 cells on the coarsest (one warp, or the
CTA), one and several pre- and post-sweeps, V- and F-cycles, axes that stop
coarsening early.  The FP32 cycle takes the same path; its distance from the
FP64 result is bounded by the rounding of a few hundred dependent operations.
"""
import numpy as np
import pytest

from hfps import workloads

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]

CASES = [
    # shape, smoother (0 red-black, 1 Chebyshev), cycle, pre, post, minimum coarse extent
    ((11, 31, 3), 1, 1, 1, 2, 3),    # 1023 cells: the finest level itself
    ((8, 8, 16), 1, 1, 1, 2, 3),     # 1024 cells: the next level down
    ((8, 16, 8), 0, 0, 2, 2, 3),
    ((20, 41, 19), 1, 1, 2, 3, 3),
    ((20, 41, 19), 0, 1, 1, 1, 3),
    ((25, 18, 33), 1, 0, 3, 1, 5),   # coarsest 4 x 5 x 5: more than a warp
    ((25, 18, 33), 0, 1, 2, 2, 9),   # coarsest 7 x 9 x 9
    ((64, 6, 5), 1, 1, 1, 1, 3),     # two axes stop early
    ((5, 4, 4), 1, 1, 1, 2, 3),      # two levels, the coarsest of 18 cells or fewer
]


@pytest.mark.parametrize("shape,smoother,cycle,pre,post,extent", CASES)
def test_small_levels_match_restatement(cuda_library, shape, smoother, cycle, pre, post, extent):
    import c_oracle
    import hfps
    import ref_oracle
    s = workloads.make("sphere64", n=shape, seed=5)
    # grids this far from cubes have no strong axis under this threshold
    policy = hfps.Policy.production().replace(
        point_smoother=smoother, cycle=cycle, pre_sweeps=pre, post_sweeps=post,
        minimum_coarse_extent=extent, anisotropy_threshold=1e3)
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=smoother, cycle=cycle, pre=pre, post=post,
                               min_coarse_extent=extent, anisotropy_threshold=1e3,
                               diagonal_shortcut=0.1), unit_linear=True)
    g = hfps.PressureSolver.from_system(s, policy)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    assert np.array_equal(g.apply_preconditioner(r), expected)
    assert np.array_equal(g.apply_preconditioner(r), expected)
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= 100 * 2.0 ** -24 * np.linalg.norm(expected)
