"""Tables shared by a process's engines (akvisqol_b200/csrc/shared_tables.h):
an engine that forms one does not hold up an engine that asks for another."""

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "native" / "shared_tables.cpp"
EXE = ROOT / "tests" / "native" / "build" / "shared_tables"


def test_properties():
    EXE.parent.mkdir(parents=True, exist_ok=True)
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", str(EXE), str(SRC), "-lpthread"], check=True)
    got = subprocess.run([str(EXE)], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0
    assert got.stdout.splitlines() == ["side by side", "formed 1, shared", "formed 2"]
