"""How the RHS group's marching kernels are split (the functions that the
launches call, compiled for the host): small boxes take one step a thread, and
the long boxes of test_flux_tiles_gpu take several in every direction, with a
shorter last segment, so that its rings wrap and its remainders are run."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from tests.test_flux_tiles_gpu import LONG, SIZES, SMS

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "steps_host.cu")
OUT = os.path.join(HERE, "_build", "libsteps.so")
CSRC = os.path.join(os.path.dirname(HERE), "asterx_b200", "csrc")


@pytest.fixture(scope="module")
def steps():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    deps = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(("cuh", "hxx"))]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                        "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC", SRC, "-o",
                        OUT], check=True)
    lib = C.CDLL(OUT)

    def of(n, te=1):
        out = (C.c_int * 3)()
        lib.rhs_steps((C.c_int * 3)(*n), te, SMS, out)
        return tuple(out)

    return of


@pytest.mark.parametrize("n", LONG)
def test_long_boxes_march(steps, n):
    for axis, s in zip((1, 2, 2), steps(n)):
        # more steps than the five slots of the ring, and a remainder
        assert s >= 6 and n[axis] % s != 0, (n, axis, s)


def test_split_by_size(steps):
    assert all(steps(n) == (1, 1, 1) for n in SIZES)
    for edge in (16, 48, 128, 256, 384):
        s = steps((edge,) * 3)
        assert all(1 <= q <= 32 for q in s)
        assert (min(s) >= 6) == (edge >= 128)
    assert steps((4, 4, 65536))[1] > 1  # grid.z stays within 65535 blocks
