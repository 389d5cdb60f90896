"""The tabulated EOS's pressure and temperature queries started from a guess
of the temperature cell (CPU, the device functions compiled as host code): any
guess gives the bits of the full search, inside and outside the table, and on
tables whose ln eps is not monotonic (where no guess is taken).  The face
state's combined query gives what the separate ones give: eps and press to the
bit, cs^2 within the rounding of the inversion it leaves out (a few ulps of
ln eps, 1e-15 of values up to 4, over the smallest slope of ln eps in ln T, 0.2
here, times the table's slope of cs^2, below 1: 1e-13), on every side of the
table's limits."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "tab_query_host.cu")
OUT = os.path.join(HERE, "_build", "libtab_query.so")
CSRC = os.path.join(os.path.dirname(HERE), "asterx_b200", "csrc")
_dp = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    deps = [SRC] + [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    if not os.path.exists(OUT) or any(os.path.getmtime(d) > os.path.getmtime(OUT) for d in deps):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-O2", "-shared",
                        "-Xcompiler", "-fPIC,-ffp-contract=off", SRC, "-o", OUT], check=True)
    L = C.CDLL(OUT)
    L.tab_query.argtypes = ([C.POINTER(C.c_int)] + [_dp] * 4 + [C.c_double] * 2 + [C.c_int]
                            + [C.c_double] * 3 + [C.c_int, _dp])
    L.tab_face.argtypes = ([C.POINTER(C.c_int)] + [_dp] * 4 + [C.c_double] * 2 + [C.c_int]
                           + [C.c_double] * 3 + [_dp])
    L.tab_face.restype = None
    return L


def _table(n, seed, noise):
    """ln P, ln(eps + shift), s, cs^2 per node, eps rising with T up to noise."""
    rng = np.random.default_rng(seed)
    lr, lt = np.linspace(-20.0, -5.0, n[0]), np.linspace(-3.0, 3.0, n[1])
    ye = np.linspace(0.05, 0.6, n[2])
    Y, T, R = np.meshgrid(ye, lt, lr, indexing="ij")
    t = np.zeros((n[2], n[1], n[0], 4))
    t[..., 0] = R + T + 0.1 * Y + 0.05 * rng.uniform(-1, 1, T.shape)
    t[..., 1] = 0.8 * T + 0.02 * R + 0.3 * Y + noise * rng.uniform(-1, 1, T.shape)
    t[..., 2], t[..., 3] = T - R, 0.3 + 0.05 * T + 0.01 * rng.uniform(-1, 1, T.shape)
    return lr, lt, ye, np.ascontiguousarray(t.reshape(-1))


@pytest.mark.parametrize("n,noise", [((6, 12, 4), 0.0), ((2, 2, 2), 0.0), ((3, 3, 2), 0.0),
                                     ((5, 40, 3), 0.02), ((5, 16, 3), 1.0)])
def test_any_hint_gives_the_full_search(lib, n, noise):
    lr, lt, ye, y = _table(n, 3 + n[1], noise)
    le = y.reshape(n[2], n[1], n[0], 4)[..., 1]
    mono = int((np.diff(le, axis=1) > 1e-12 * np.abs(le).max()).all())
    assert mono == (noise < 0.5)
    nn = (C.c_int * 3)(*n)
    ptr = [a.ctypes.data_as(_dp) for a in (lr, lt, ye, y)]
    rng = np.random.default_rng(17)

    def query(rho, eps, yq, hint):
        out = np.zeros(4)
        h = lib.tab_query(nn, *ptr, 0.01, 1e-3, mono, rho, eps, yq, hint,
                          out.ctypes.data_as(_dp))
        return out, h

    inside = 0
    for _ in range(300):
        rho = np.exp(rng.uniform(-21, -4))
        eps = np.exp(rng.uniform(le.min() - 0.3, le.max() + 0.3)) - 0.01
        yq = rng.uniform(0.0, 0.7)  # not clamped by the queries
        want, cell = query(rho, eps, yq, -1)
        inside += 0 <= cell < n[1]
        for hint in range(-2, n[1] + 2):
            got, _ = query(rho, eps, yq, hint)
            assert got.tobytes() == want.tobytes(), (rho, eps, yq, hint, got, want)
    assert inside > 50


@pytest.mark.parametrize("n,noise", [((6, 12, 4), 0.0), ((2, 2, 2), 0.0), ((5, 40, 3), 0.02),
                                     ((5, 16, 3), 1.0)])
@pytest.mark.parametrize("shift", [0.0, 0.01])
def test_face_state_is_the_separate_queries(lib, n, noise, shift):
    lr, lt, ye, y = _table(n, 3 + n[1], noise)
    le = y.reshape(n[2], n[1], n[0], 4)[..., 1]
    mono = int((np.diff(le, axis=1) > 1e-12 * np.abs(le).max()).all())
    nn = (C.c_int * 3)(*n)
    ptr = [a.ctypes.data_as(_dp) for a in (lr, lt, ye, y)]
    rng = np.random.default_rng(19)
    for _ in range(2000):
        rho, temp = np.exp(rng.uniform(-21, -4)), np.exp(rng.uniform(-3.3, 3.3))
        out = np.zeros(8)
        lib.tab_face(nn, *ptr, shift, 0.1, mono, rho, temp, rng.uniform(0.0, 0.7),
                     out.ctypes.data_as(_dp))
        assert out[[0, 1, 3]].tobytes() == out[[4, 5, 7]].tobytes(), (rho, temp, out)
        assert abs(out[2] - out[6]) <= (1e-13 if mono else 0.0), (rho, temp, out)
