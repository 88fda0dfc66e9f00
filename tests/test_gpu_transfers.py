"""Transfers with all three axes coarsened (a thread per fine cell in the
restriction, 2x2x2 fine cells per thread in the prolongation) and the flat
multigrid entry and exit, bit for bit the C restatement's: rows that end inside,
at and past a block's 32 coarse cells, odd and even extents per axis, both point
smoothers, and the residual-minimising exit."""
import numpy as np
import pytest

from hfps import workloads

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]


@pytest.mark.parametrize("shape", [(64, 17, 16), (65, 12, 18), (130, 9, 11), (63, 18, 13),
                                   (12, 40, 33)])
@pytest.mark.parametrize("smoother", [0, 1])
def test_point_transfers_match_restatement(cuda_library, shape, smoother):
    import c_oracle
    import hfps
    import ref_oracle
    s = workloads.make("sphere64", n=shape, seed=6)
    policy = hfps.Policy.production().replace(point_smoother=smoother, anisotropy_threshold=1e3)
    mg = ref_oracle.MgPolicy(smoother=smoother, cycle=1, pre=1, post=2, diagonal_shortcut=0.1,
                             anisotropy_threshold=1e3)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    for unit in (1, 0):
        oracle = c_oracle.OracleSession(s, mg, unit_linear=bool(unit))
        z = hfps.PressureSolver.from_system(s, policy.replace(unit_linear=unit)) \
            .apply_preconditioner(r)
        expected = oracle.apply_mg(r)
        if unit:
            assert np.array_equal(z, expected)
        else:
            # the scale is a quotient of two sums, added in another order here
            assert np.linalg.norm(z - expected) <= 4 * np.sqrt(s.cells) * 2.0 ** -53 \
                * np.linalg.norm(expected)


@pytest.mark.parametrize("shape,post", [((9, 9, 9), 1), ((33, 18, 21), 1), ((48, 50, 54), 3),
                                        ((51, 51, 52), 1)])
@pytest.mark.parametrize("smoother", [0, 1])
def test_prolongation_with_first_step_matches_restatement(cuda_library, shape, post, smoother):
    """One and three post-smoothing steps (the first of them taken with the
    prolongation up to 2^17 cells), cells at, inside and past a block's 8 x 8 x 4,
    and a grid just above that size."""
    import c_oracle
    import hfps
    import ref_oracle
    s = workloads.make("sphere64", n=shape, seed=6)
    policy = hfps.Policy.production().replace(point_smoother=smoother, post_sweeps=post,
                                              anisotropy_threshold=1e3)
    mg = ref_oracle.MgPolicy(smoother=smoother, cycle=1, pre=1, post=post, diagonal_shortcut=0.1,
                             anisotropy_threshold=1e3)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    z = hfps.PressureSolver.from_system(s, policy).apply_preconditioner(r)
    oracle = c_oracle.OracleSession(s, mg, unit_linear=True)
    assert np.array_equal(z, oracle.apply_mg(r))


@pytest.mark.parametrize("shape,mixed_bar", [((125, 249, 121), 1e-5), ((64, 63, 468), 1e-4)])
@pytest.mark.parametrize("pre,post", [(3, 1), (1, 3)])
def test_tiled_stages_match_restatement(cuda_library, shape, mixed_bar, pre, post):
    """FP32 Chebyshev stages over 3-D tiles, on levels that fill three quarters of
    a wave of them: tiles cut in every direction, and the first, middle and last
    stage and the only one.  FP64 stages are flat and equal bit for bit.  A FP32
    diagonal is rounded apart from its faces, which adds or takes up to u of it and
    so moves the smoothest mode along n cells by up to u n^2 4 / pi^2 (1.5e-3 and
    5.3e-3 here); the roundings are of either sign, and the bars are four times the
    distance measured, 2.3e-6 and 2.5e-5."""
    import c_oracle
    import hfps
    import ref_oracle
    s = workloads.make("sphere64", n=shape, seed=6)
    policy = hfps.Policy.production().replace(pre_sweeps=pre, post_sweeps=post,
                                              anisotropy_threshold=1e3)
    mg = ref_oracle.MgPolicy(smoother=1, cycle=1, pre=pre, post=post, diagonal_shortcut=0.1,
                             anisotropy_threshold=1e3)
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    g = hfps.PressureSolver.from_system(s, policy)
    expected = c_oracle.OracleSession(s, mg, unit_linear=True).apply_mg(r)
    assert np.array_equal(g.apply_preconditioner(r), expected)
    mixed = g.apply_preconditioner(r, precision=hfps.MIXED)
    assert np.linalg.norm(mixed - expected) <= mixed_bar * np.linalg.norm(expected)
