"""Line levels in the one-CTA launch of the smallest levels (kernels_small.cu)
and the dense coarsest map of several line axes, against the C restatement:
lines of one cell up to the 32 a warp holds and of 33 (left to the launches
above), one, two and three strong axes, V- and F-cycles, unit and several
sweeps, and a finest level that is itself small.  The bar is the line
relaxation's, 1e-11 relative in FP64 (exact eliminations and sums in another
order).  An FP32 elimination is off by the unit roundoff times the condition of
its line, up to the square of the line's cells for the smooth modes a random
rhs holds."""
import numpy as np
import pytest

from hfps import workloads
from test_gpu_parity import stretched_front

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]

CASES = [
    # shape, stretched axis, threshold, strong axes, cycle, pre, post
    ((27, 32, 23), 1, 4.0, 2, 1, 1, 2),
    ((27, 33, 23), 1, 4.0, 2, 1, 1, 2),
    ((30, 21, 26), 2, 4.0, 4, 0, 2, 1),
    ((17, 40, 41), 0, 4.0, 1, 1, 2, 2),
    ((9, 10, 11), 1, 4.0, 2, 1, 1, 1),     # 990 cells: the finest level
    ((60, 40, 12), 1, 3.0, 3, 1, 1, 2),    # x and y strong, full coarsening
    ((60, 40, 12), 1, 3.0, 3, 0, 2, 2),
    ((40, 24, 20), 0, 1.1, 3, 1, 1, 2),
]


@pytest.mark.parametrize("shape,axis,threshold,strong,cycle,pre,post", CASES)
def test_small_line_levels_match_restatement(cuda_library, shape, axis, threshold, strong, cycle,
                                             pre, post):
    import c_oracle
    import hfps
    import ref_oracle
    s = stretched_front(shape, axis, 1.0 + 3.0 / shape[axis])
    policy = hfps.Policy.production().replace(cycle=cycle, pre_sweeps=pre, post_sweeps=post,
                                              anisotropy_threshold=threshold)
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=1, cycle=cycle, pre=pre, post=post, diagonal_shortcut=0.1,
                               anisotropy_threshold=threshold), unit_linear=True, line_order=1)
    g = hfps.PressureSolver.from_system(s, policy)
    assert g.levels()[0][3] == strong
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    size = np.linalg.norm(expected)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= 1e-11 * size
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= max(shape) ** 2 * 2.0 ** -24 * size
