"""The coalesced chunked scan of x-lines (k_line_scan_x) against the C
restatement: rows that are no multiple of a chunk or a warp, odd transverse
extents (a colour of fewer lines on every other plane), several lines per
block and one, with and without a second line axis.  The bar is the line
relaxation's (exact eliminations in another order): 1e-11 relative in FP64, and for
the longest lines a sixteenth of the unit roundoff times their condition, the square
of their cells (2.9e-11 at 2048; measured 9.6e-12).  FP32 adds the rounding of the
coefficients, which the condition amplifies case by case: its bars are four times
the distance measured, and never above the roundoff times the square of the cells."""
import numpy as np
import pytest

from hfps import workloads
from test_gpu_parity import stretched_front

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]


@pytest.mark.parametrize("shape,both,mixed_bar", [
    ((33, 64, 40), False, 1.1e-5), ((100, 37, 61), False, 6.0e-4), ((257, 48, 48), False, 1.6e-3),
    ((71, 66, 63), True, 3.5e-5),
    # several warps per line: 2 to 8 of them, up to the longest line
    ((520, 32, 33), False, 8.5e-3), ((700, 33, 32), False, 5.5e-3),
    ((1030, 24, 46), False, 1.1e-2), ((2048, 32, 32), False, 2.0e-2)])
def test_x_lines_match_restatement(cuda_library, shape, both, mixed_bar):
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
    bar = max(1e-11, shape[0] ** 2 * 2.0 ** -53 / 16)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= bar * size
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= mixed_bar * size
