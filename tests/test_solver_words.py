"""The solver's packed words at the ends of their fields' ranges.

csrc/solver_words.cuh compiles as plain C++; tests/words/check_words.cpp packs and reads
back every field where it is widest: a body's joint rows and finished joints up to the
joints that solve_flow takes, a colouring claim's contact index above 2^24, and the point
slots of the most contacts a world has room for."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "physecs_gb300", "csrc")


def test_fields_hold_their_ranges(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "check_words")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(HERE, "words", "check_words.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
