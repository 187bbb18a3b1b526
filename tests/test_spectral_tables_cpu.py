"""The FMA forms' spectral energies (akvisqol_b200/csrc/spectral_tables.cpp)
on the CPU: sum |X|^2 G less the squared tail functionals against the cascade
run sample by sample, both in extended precision, so that what is left is the
tables' own error. It stays below the f64 recurrence's rounding (up to 3.5e-13
of a band's RMS): 2e-13."""

import ctypes
import subprocess
from ctypes import POINTER, c_double, c_int, c_size_t, c_uint32
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "native" / "spectral_shim.cpp"
LIB = ROOT / "tests" / "native" / "build" / "libspectral_shim.so"


@pytest.fixture(scope="module")
def shim():
    LIB.parent.mkdir(parents=True, exist_ok=True)
    csrc = ROOT / "akvisqol_b200" / "csrc"
    srcs = [SRC, csrc / "spectral_tables.cpp", csrc / "host_model.cpp", csrc / "lattice.cpp", csrc / "tflite.cpp"]
    if not LIB.is_file() or any(s.stat().st_mtime > LIB.stat().st_mtime for s in srcs):
        model = ROOT / "akvisqol_b200" / "model" / "libsvm_nu_svr_model.txt"
        lattice = next((ROOT / "akvisqol_b200" / "model").glob("lattice_*.tflite"))
        subprocess.run(["g++", "-std=c++17", "-O2", "-march=x86-64-v3", "-fPIC", "-shared", "-ffp-contract=off",
                        "-I/usr/local/cuda/include", f"-DVQB_MODEL_PATH={model}", f"-DVQB_LATTICE_PATH={lattice}",
                        "-o", str(LIB)] + [str(s) for s in srcs] + ["-lpthread"], check=True)
    lib = ctypes.CDLL(str(LIB))
    D = POINTER(c_double)
    lib.ss_frame.restype = c_int
    lib.ss_frame.argtypes = [c_size_t, c_uint32, c_double, D, c_size_t, D, D]
    return lib


def frame_of(kind, n):
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.standard_normal(n)) * 0.01 + 0.1 * rng.standard_normal(n)
    if kind == "onset":  # nearly all of the low bands' energy behind the frame
        x[: n - n // 16] = 0.0
    elif kind == "tone":  # bands far from it hold its leakage alone
        x = np.sin(2 * np.pi * 0.21 * np.arange(n))
    return x


@pytest.mark.parametrize("kind", ["noise", "onset", "tone"])
@pytest.mark.parametrize("nb,rate", [(32, 48000), (32, 44100), (32, 22050), (21, 16000), (32, 8000), (32, 6420), (32, 51200)])
def test_energies(shim, nb, rate, kind):
    window = int(np.floor(rate * 0.08 + 0.5))
    high = min(8000.0, rate / 2) if nb == 21 else rate / 2
    x = frame_of(kind, window)
    got, want = np.zeros(nb), np.zeros(nb)
    D = POINTER(c_double)
    p = lambda a: a.ctypes.data_as(D)  # noqa: E731
    assert shim.ss_frame(nb, rate, high, p(x), window, p(got), p(want)) == 1
    # cells under 1e-9 of the frame's largest energy are floored before they are used
    heard = want > 3e-5 * want.max()
    assert heard.any()
    assert np.max(np.abs(got - want)[heard] / want[heard]) <= 2e-13


def test_other_windows_keep_the_recurrence(shim):
    for window in (16, 512, 4097, 7680):
        x = np.zeros(window)
        z = np.zeros(32)
        D = POINTER(c_double)
        assert shim.ss_frame(32, 48000, 24000.0, x.ctypes.data_as(D), window, z.ctypes.data_as(D), z.ctypes.data_as(D)) == 0
