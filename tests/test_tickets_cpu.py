"""The arithmetic that places a ticket in a job (csrc/tickets.h), compiled for the host."""
import ctypes
import os
import random
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no C++ compiler"
    d = tmp_path_factory.mktemp("tickets")
    src = d / "t.cpp"
    src.write_text('#include "tickets.h"\nextern "C" unsigned place(unsigned g, unsigned n, int* s, unsigned* f) { return ofa::place_ticket(g, n, *s, *f); }\n')
    lib = d / "t.so"
    subprocess.run([cxx, "-O1", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "open-flapping-airplanes_b200", "csrc"), "-o", str(lib), str(src)], check=True)
    f = ctypes.CDLL(str(lib)).place
    f.restype, f.argtypes = ctypes.c_uint, [ctypes.c_uint, ctypes.c_uint, ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_uint)]
    return f


@pytest.mark.parametrize("per_step", [2, 3, 299, 3936, 57946, 1 << 24, (1 << 31) - 1])
@pytest.mark.parametrize("late", [0, 1, 2 ** 31 - 1, 2 ** 31, 2 ** 31 + 5, 3_999_990_000])
def test_a_block_finds_its_tickets_wherever_its_first_one_lies(place, per_step, late):
    rng = random.Random(per_step + late)
    step, first, g = ctypes.c_int(0), ctypes.c_uint(0), late
    for _ in range(200):
        r = place(g, per_step, step, first)
        assert (step.value, r) == divmod(g, per_step) and first.value == g - r
        g += rng.choice([1, 7, 296, per_step - 1, per_step, per_step + 1, 2 * per_step, 5 * per_step + 1])
        if g >= 4_000_000_000:
            break
