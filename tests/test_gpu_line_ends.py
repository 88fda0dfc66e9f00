"""Line levels whose Neumann boundary faces are not zero keep the end terms of
their lines (the cell reads itself through the face); with zero faces, as
set_beta and assemble make them, the passes leave them out.  Both against the C
restatement at the line relaxation's bar, 1e-11 relative."""
import numpy as np
import pytest

from hfps import workloads
from test_gpu_parity import stretched_front

pytestmark = [pytest.mark.gpu, pytest.mark.usefixtures("oracle_built")]


# The kernel without end terms serves y-lines in split rows whose blocks then take
# fewer waves: 101x150x99 has 5049 lines a colour, 8 a block of 3 warps, 632 blocks
# where 592 are resident with end terms and 740 without; 131x256x67 has 4422, 553
# blocks of 4 warps, 444 and 592.  The other grids keep the kernel with the end terms.
@pytest.mark.parametrize("shape,axis", [
    ((60, 48, 48), 0), ((48, 60, 48), 1), ((48, 48, 60), 2),
    ((101, 150, 99), 1), ((131, 256, 67), 1), ((131, 133, 160), 2)])
@pytest.mark.parametrize("face", [0.0, 0.3])
def test_neumann_faces_at_line_ends(cuda_library, shape, axis, face):
    import c_oracle
    import hfps
    import ref_oracle
    s = stretched_front(shape, axis, 1.0 + 3.6 / shape[axis])
    for f, dim in ((s.face_x, 2), (s.face_y, 1), (s.face_z, 0)):
        low = [slice(None)] * 3
        low[dim] = 0
        f[tuple(low)] = face * f.max()
        s.diagonal[tuple(low)] += f[tuple(low)]
    oracle = c_oracle.OracleSession(
        s, ref_oracle.MgPolicy(smoother=1, cycle=1, pre=1, post=2, diagonal_shortcut=0.1),
        unit_linear=True, line_order=1)
    g = hfps.PressureSolver.from_system(s, hfps.Policy.production())
    assert g.levels()[0][3] == 1 << axis
    r = np.ascontiguousarray(workloads.normals(3, s.cells).reshape(s.rhs.shape))
    expected = oracle.apply_mg(r)
    assert np.linalg.norm(g.apply_preconditioner(r) - expected) <= 1e-11 * np.linalg.norm(expected)
