"""A process that cannot start threads gets its results from fewer of them, or
an exception, never std::terminate: tests/native/thread_failure.cpp with a
pthread_create that refuses all but the first few."""

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "native" / "thread_failure.cpp"
EXE = ROOT / "tests" / "native" / "build" / "thread_failure"


@pytest.fixture(scope="module")
def run():
    EXE.parent.mkdir(parents=True, exist_ok=True)
    csrc = ROOT / "akvisqol_b200" / "csrc"
    srcs = [SRC, csrc / "spectral_tables.cpp", csrc / "host_model.cpp", csrc / "lattice.cpp", csrc / "tflite.cpp"]
    headers = [csrc / "threads.h", csrc / "spectral_tables.h"]
    if not EXE.is_file() or any(s.stat().st_mtime > EXE.stat().st_mtime for s in srcs + headers):
        model = ROOT / "akvisqol_b200" / "model" / "libsvm_nu_svr_model.txt"
        lattice = next((ROOT / "akvisqol_b200" / "model").glob("lattice_*.tflite"))
        subprocess.run(["g++", "-std=c++17", "-O2", "-march=x86-64-v3", "-ffp-contract=off", "-rdynamic",
                        "-I/usr/local/cuda/include", f"-DVQB_MODEL_PATH={model}", f"-DVQB_LATTICE_PATH={lattice}",
                        "-o", str(EXE)] + [str(s) for s in srcs] + ["-lpthread", "-ldl"], check=True)
    return lambda threads: subprocess.run([str(EXE), str(threads)], capture_output=True, text=True, timeout=120)


@pytest.fixture(scope="module")
def all_threads(run):
    got = run(1000)
    assert got.returncode == 0 and got.stdout.split()[1:] == ["499500", "caught"], got
    return got.stdout


@pytest.mark.parametrize("threads", [0, 1, 3])
def test_threads_that_cannot_start(run, all_threads, threads):
    got = run(threads)
    assert got.returncode == 0, got
    assert got.stdout == all_threads
