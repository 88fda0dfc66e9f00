"""Calls on device arrays used in place against the same calls through the
staging vectors (host arrays): outputs that overlap the input in every way, an
output that is the input, slices at odd offsets of a larger buffer, changing
vectors on one captured multigrid graph, and the graph kept across coefficient
updates.  All of it bit for bit."""
import numpy as np
import pytest

from hfps import workloads

pytestmark = pytest.mark.gpu


def system(seed=3):
    return workloads.make("wrinkled256", n=(20, 24, 18), stretch_y=1.1, seed=seed)


@pytest.mark.parametrize("call", ["operator", "mg", "mixed", "ic0"])
@pytest.mark.parametrize("shift", [-7, 0, 1, 5000, None])
def test_overlapping_and_offset_arrays(cuda_library, call, shift):
    import hfps
    import torch
    s = system()
    policy = hfps.Policy.production()
    if call == "ic0":
        policy = policy.replace(preconditioner=hfps.IC0)
    g = hfps.PressureSolver.from_system(s, policy)
    n = s.cells
    v = workloads.normals(5, n)

    def apply(a, out):
        if call == "operator":
            return g.apply_operator(a, out=out)
        return g.apply_preconditioner(a, out=out,
                                      precision=hfps.MIXED if call == "mixed" else hfps.FP64)

    expected = apply(v, np.empty_like(v))
    buffer = torch.zeros(3 * n + 64, dtype=torch.float64, device="cuda")
    at = n + 9
    x = buffer[at:at + n]
    x.copy_(torch.from_numpy(v))
    out = buffer[2 * n + 11:3 * n + 11] if shift is None else buffer[at + shift:at + shift + n]
    apply(x, out)
    assert np.array_equal(out.cpu().numpy(), expected)


@pytest.mark.parametrize("unit", [0, 1])
def test_one_graph_serves_every_vector_and_update(cuda_library, unit):
    """Vectors change from call to call, precisions alternate, coefficients are
    replaced in between: each result is a fresh solver's."""
    import hfps
    import torch

    def device(a):
        return torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()

    systems = [system(3), system(4)]
    systems[1].face_x *= 1.5
    systems[1].diagonal += (systems[1].face_x[:, :, :-1] + systems[1].face_x[:, :, 1:]) / 3.0
    policy = hfps.Policy.production().replace(unit_linear=unit)
    kept = hfps.PressureSolver.from_system(systems[0], policy)
    vectors = [device(workloads.normals(k, systems[0].cells)) for k in range(3)]
    for turn in range(2):
        for s in systems:
            kept.set_coefficients(s.diagonal, s.face_x, s.face_y, s.face_z)
            for precision in (hfps.FP64, hfps.MIXED):
                for v in vectors:
                    z = kept.apply_preconditioner(v, precision=precision)
                    fresh = hfps.PressureSolver.from_system(s, policy)
                    assert torch.equal(z, fresh.apply_preconditioner(v, precision=precision))
                    fresh.close()
            if turn == 0:
                options = dict(algorithm=hfps.FGMRES, restart=5, rtol=1e-9)
                x, info = kept.solve(device(s.rhs), **options)
                fresh = hfps.PressureSolver.from_system(s, policy)
                y, other = fresh.solve(device(s.rhs), **options)
                assert torch.equal(x, y) and info["iterations"] == other["iterations"]
                fresh.close()
