"""Host paths of the library that no GPU run reaches: calls that the CUDA
runtime refuses, and what several handles in one process do to one another.
The library runs here on a stand-in for the runtime (fake_cudart.cpp), each
case in a process of its own; kernels do not run, so no result is looked at."""
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"

PREAMBLE = """
import ctypes, sys
import numpy as np
sys.path.insert(0, {package!r})
import hfps
fake = ctypes.CDLL({fake!r})
fake.fake_entry_argument.restype = ctypes.c_void_p

def solver(shape, stretch=None, **policy):
    faces = []
    for axis, n in enumerate(shape):
        w = (1.0 + 5.0 / n if axis == stretch else 1.0) ** np.arange(n)
        faces.append(np.concatenate([[0.0], np.cumsum(w * n / w.sum())]))
    policy.setdefault("anisotropy_threshold", 1e9 if stretch is None else 4.0)
    s = hfps.PressureSolver(shape, faces, (1, 0, 1, 1, 1, 1), None,
                            hfps.Policy.production().replace(**policy))
    update(s)
    return s

def update(s):
    s.set_coefficients(np.ones(s.cells), *(np.ones(n) for n in s.face_counts))

def apply(s, r=None, precision=hfps.FP64, z=None):
    r = np.ones(s.cells) if r is None else r
    z = np.empty(s.cells) if z is None else z
    s._check(s._lib.hfps_apply_preconditioner(s._handle, r.ctypes.data, z.ctypes.data,
                                              hfps.DEVICE, precision), "apply")

def refused(call):
    try:
        call()
    except hfps.SolverError as e:
        return str(e)
    return ""
"""


@pytest.fixture(scope="module")
def run(cuda_library, tmp_path_factory):
    if not os.path.isdir(CUDA_INCLUDE):
        pytest.skip("CUDA headers not installed")
    fake = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CUDA_INCLUDE}",
                    os.path.join(HERE, "fake_cudart.cpp"), "-o", fake], check=True)
    preamble = PREAMBLE.format(package=os.path.dirname(cuda_library), fake=fake)

    def run(body):
        proc = subprocess.run([sys.executable, "-c", preamble + textwrap.dedent(body)],
                              env=dict(os.environ, LD_PRELOAD=fake), capture_output=True,
                              text=True, timeout=300)
        assert proc.returncode == 0, proc.stdout + proc.stderr
    return run


@pytest.mark.parametrize("first,second,stretch", [
    ((40, 40, 40), (72, 72, 72), None),    # one-CTA point levels: 86,112 and 67,248 bytes
    ((512, 40, 40), (600, 40, 40), 0),     # x-line scan: 56,320 and 50,160
    ((40, 500, 40), (40, 450, 40), 1),     # sweeps of a coarsest level of y-lines
])
def test_shared_memory_limits_hold_for_every_handle(run, first, second, stretch):
    """A kernel's limit belongs to the process: a second handle, whose launches
    need less, must not take it below what the first one's need."""
    run(f"""
    a = solver({first}, {stretch})
    b = solver({second}, {stretch})
    for s in (a, b, a):
        for precision in (hfps.FP64, hfps.MIXED):
            apply(s, precision=precision)
        update(s)
    assert fake.fake_calls(b"cudaFuncSetAttribute") > 0
    assert fake.fake_lowered() == 0
    """)


@pytest.mark.parametrize("call", ["apply", "update", "flux"])
@pytest.mark.parametrize("shape,stretch", [((40, 40, 40), None), ((60, 24, 20), 0)])
def test_refused_launch_is_reported(run, call, shape, stretch):
    """Whichever launch of a call the runtime refuses, the call says so, no
    graph that lacks the kernel is kept, and the next call is whole again."""
    run(f"""
    s = solver({shape}, {stretch})
    c = [np.ones(n) for n in s.face_counts]
    calls = {{"apply": lambda: apply(s), "update": lambda: update(s),
              "flux": lambda: s.correct_flux(np.ones(s.cells), c, [v.copy() for v in c])}}
    call = calls[{call!r}]
    before = fake.fake_calls(b"cudaLaunchKernelExC")
    call()
    launches = fake.fake_calls(b"cudaLaunchKernelExC") - before
    whole = fake.fake_launched(b"k_")
    assert launches > 0 and (whole == launches or {call!r} != "apply")
    for nth in range(1, launches + 1):
        if {call!r} == "apply":
            s = solver({shape}, {stretch})
        graphs = fake.fake_calls(b"cudaGraphLaunch")
        fake.fake_fail(b"cudaLaunchKernelExC", nth)
        assert refused(call), nth
        assert fake.fake_calls(b"cudaGraphLaunch") == graphs
        call()
        assert fake.fake_launched(b"k_") == whole
    """)


@pytest.mark.parametrize("unit", [1, 0])
def test_graph_serves_the_vectors_of_its_call(run, unit):
    """One captured application serves every pair of vectors: after an update
    of its nodes that failed half-way, and where the capture could not tell
    which nodes they are (then it is captured anew for another pair)."""
    run(f"""
    def pair(s):
        return np.ones(s.cells), np.empty(s.cells)

    def solve_on(s, v):
        apply(s, v[0], z=v[1])
        return fake.fake_entry_argument()

    s = solver((20, 20, 20), unit_linear={unit})
    first, second = pair(s), pair(s)
    solve_on(s, first)
    assert solve_on(s, second) == second[0].ctypes.data
    for nth in range(1, 3 if {unit} else 4):
        fake.fake_fail(b"cudaGraphExecKernelNodeSetParams", nth)
        assert refused(lambda: solve_on(s, first)), nth
        assert solve_on(s, second) == second[0].ctypes.data, nth
    for nth in range(1, 3 if {unit} else 4):
        s = solver((20, 20, 20), unit_linear={unit})
        fake.fake_fail(b"cudaStreamGetCaptureInfo_v3", nth)
        captures = fake.fake_calls(b"cudaStreamBeginCapture")
        solve_on(s, first)
        solve_on(s, first)
        assert fake.fake_calls(b"cudaStreamBeginCapture") == captures + 1
        solve_on(s, second)
        assert fake.fake_calls(b"cudaStreamBeginCapture") == captures + 2, nth
    """)


@pytest.mark.parametrize("preconditioner,stretch", [("IC0", None), ("MG", None), ("MG", 1)])
def test_failed_update_leaves_no_coefficients(run, preconditioner, stretch):
    """An update that ends with any error (a refused launch, or one of the
    synchronisations that read what it found; the IC(0) factorisation's are the
    last) leaves no levels or pivots that a later call could run on; the next
    update does."""
    run(f"""
    s = solver((20, 30, 20), {stretch}, preconditioner=hfps.solver.{preconditioner})
    for name in (b"cudaStreamSynchronize", b"cudaLaunchKernelExC"):
        before = fake.fake_calls(name)
        update(s)
        for nth in range(1, fake.fake_calls(name) - before + 1):
            fake.fake_fail(name, nth)
            assert refused(lambda: update(s))
            assert "coefficients not set" in refused(lambda: apply(s)), (name, nth)
            update(s)
            apply(s)
    """)


@pytest.mark.parametrize("shape", [(2, 600000, 1), (1, 2, 600000), (600000, 2, 1)])
@pytest.mark.parametrize("smoother", [0, 1])
def test_long_grids_are_within_launch_limits(run, shape, smoother):
    """Launch shapes of grids that are long in one direction: the second and
    third grid dimension hold 65535 blocks each."""
    run(f"""
    s = solver({shape}, point_smoother={smoother})
    for precision in (hfps.FP64, hfps.MIXED):
        apply(s, precision=precision)
    """)
