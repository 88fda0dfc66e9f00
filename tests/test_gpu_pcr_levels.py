"""Line levels relaxed with PCR, against the C restatement's zebra order: rows of
every power of two up to 256 and just past one, exchanged within a warp (up to 32
rows) and across warps, and numbers of lines at and past what one cluster launch
of all passes holds, along each axis.  The bars are those of the line relaxation:
1e-11 relative in FP64 (exact eliminations in another order), and in FP32 an
eighth of the unit roundoff times the square of the line's rows, the condition of
its smoothest modes (measured 1/30 of that product at 64 to 256 rows, 1/14 at
most)."""
import numpy as np
import pytest

from hfps import workloads
from test_gpu_parity import stretched_front

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]

CASES = [
    # line axis, rows, the other two extents (lower axis first)
    (1, 16, (16, 16)),    # 128 lines a colour: 8 CTAs of 16
    (1, 16, (17, 16)),    # 144: separate passes
    (1, 17, (16, 8)),     # 64 lines of 32 threads
    (1, 32, (9, 15)),     # separate passes
    (1, 33, (8, 8)),      # first with shared memory
    (1, 64, (7, 9)),
    (1, 129, (4, 4)),
    (1, 256, (4, 4)),
    (1, 256, (4, 5)),     # separate passes
    (0, 30, (11, 10)),
    (0, 100, (6, 5)),
    (2, 24, (12, 9)),
    (2, 65, (5, 6)),
]


@pytest.mark.parametrize("axis,rows,others", CASES)
@pytest.mark.parametrize("pre,post", [(1, 2), (3, 1)])
def test_pcr_levels_match_restatement(cuda_library, axis, rows, others, pre, post):
    import c_oracle
    import hfps
    import ref_oracle
    shape = list(others)
    shape.insert(axis, rows)
    s = stretched_front(tuple(shape), axis, 1.0 + 3.0 / rows)
    policy = hfps.Policy.production().replace(pre_sweeps=pre, post_sweeps=post,
                                              anisotropy_threshold=4.0)
    g = hfps.PressureSolver.from_system(s, policy)
    assert g.levels()[0][3] == 1 << axis
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=1, cycle=1, pre=pre, post=post, diagonal_shortcut=0.1,
                               anisotropy_threshold=4.0), unit_linear=True, line_order=1)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    size = np.linalg.norm(expected)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= 1e-11 * size
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= rows ** 2 * 2.0 ** -24 / 8 * size


@pytest.mark.parametrize("axis,rows,others,extent", [
    (0, 16, (26, 26), 13), (0, 31, (18, 18), 9), (1, 32, (18, 18), 9), (2, 60, (18, 18), 9),
    (2, 64, (18, 18), 9), (1, 100, (10, 10), 5), (0, 130, (10, 10), 5), (0, 256, (10, 10), 5)])
def test_coarsest_line_levels_match_restatement(cuda_library, axis, rows, others, extent):
    """Coarsest levels of more cells than the dense map holds are swept by one
    CTA: rows that fill the threads of a line, and rows that do not."""
    import c_oracle
    import hfps
    import ref_oracle
    shape = list(others)
    shape.insert(axis, rows)
    s = stretched_front(tuple(shape), axis, 1.0 + 3.0 / rows)
    policy = hfps.Policy.production().replace(anisotropy_threshold=4.0,
                                              minimum_coarse_extent=extent)
    g = hfps.PressureSolver.from_system(s, policy)
    assert g.levels()[0][3] == 1 << axis
    assert np.prod(g.levels()[-1][:3]) > 2048
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=1, cycle=1, pre=1, post=2, diagonal_shortcut=0.1,
                               min_coarse_extent=extent, anisotropy_threshold=4.0),
        unit_linear=True, line_order=1)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= 1e-11 * np.linalg.norm(expected)
