"""The tiled IC(0) sweeps (kernels_dic.cu): one application bit for bit the C
restatement's, whose sweeps are sequential, on grids of one tile, of partial
edge tiles along y and z (tiles are 16 x 8 columns), of x extents that are no
multiple of a chunk (8 steps) or shorter than one, and of many tiles.  A NaN of
every bit pattern passes through the tile borders, where one pattern stands for
an entry that has not arrived."""
import numpy as np
import pytest

from hfps import workloads

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]


def solver(hfps, s):
    return hfps.PressureSolver.from_system(s, hfps.Policy.default().replace(
        preconditioner=hfps.IC0, anisotropy_threshold=1e3))


@pytest.mark.parametrize("shape", [
    (5, 4, 4), (7, 16, 8), (8, 17, 8), (9, 16, 9), (33, 31, 7), (64, 15, 25), (50, 50, 50)])
def test_sweeps_match_sequential_restatement(cuda_library, shape):
    import c_oracle
    import hfps
    import ref_oracle
    s = workloads.make("sphere64", n=shape, seed=2)
    oracle = c_oracle.OracleSession(s, ref_oracle.MgPolicy(anisotropy_threshold=1e3),
                                    preconditioner="dic")
    r = np.ascontiguousarray(workloads.normals(7, s.cells).reshape(s.rhs.shape))
    g = solver(hfps, s)
    for _ in range(2):
        assert np.array_equal(g.apply_preconditioner(r), oracle.apply_preconditioner(r))


@pytest.mark.parametrize("bits", [0xFFFFFFFFFFFFFFFF, 0x7FF8000000000000, 0x7FF8000000000001])
def test_nan_passes_tile_borders(cuda_library, bits):
    import hfps
    s = workloads.make("sphere64", n=(20, 40, 20), seed=2)
    r = np.array(s.rhs)
    r[2, 3, 4] = np.array([bits], dtype=np.uint64).view(np.float64)[0]
    z = solver(hfps, s).apply_preconditioner(r)
    assert np.isnan(z[2, 3, 4]) and np.isnan(z[-1, -1, -1]) and np.isnan(z[12, 35, 15])
