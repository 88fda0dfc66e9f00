"""The coalesced chunked scan of x-lines (k_line_scan_x) against the C
restatement: rows that are no multiple of a chunk or a warp, odd transverse
extents (a colour of fewer lines on every other plane), several lines per
block and one, with and without a second line axis.  The bar is the line
relaxation's (exact eliminations in another order): 1e-11 relative in FP64.  An FP32 elimination is off by the
unit roundoff times the condition of its line, up to the square of the line's
cells for the smooth modes a random rhs holds."""
import numpy as np
import pytest

from hfps import workloads
from test_gpu_parity import stretched_front

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]


@pytest.mark.parametrize("shape,both", [
    ((33, 64, 40), False), ((100, 37, 61), False), ((257, 48, 48), False),
    ((1030, 24, 46), False), ((71, 66, 63), True),
    # several warps per line: 2 to 8 of them, up to the longest line
    ((520, 32, 33), False), ((700, 33, 32), False), ((2048, 32, 32), False)])
def test_x_lines_match_restatement(cuda_library, shape, both):
    import c_oracle
    import hfps
    import ref_oracle
    s = stretched_front(shape, 0, 1.0 + 5.0 / shape[0])
    # a low threshold makes the shorter transverse axis strong as well
    threshold = 1.02 if both else 4.0
    policy = hfps.Policy.production().replace(anisotropy_threshold=threshold)
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=1, cycle=1, pre=1, post=2, diagonal_shortcut=0.1,
                               anisotropy_threshold=threshold), unit_linear=True, line_order=1)
    g = hfps.PressureSolver.from_system(s, policy)
    assert g.levels()[0][3] & 1 and (bin(g.levels()[0][3]).count("1") > 1) == both
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    size = np.linalg.norm(expected)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= 1e-11 * size
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= max(shape) ** 2 * 2.0 ** -24 * size
