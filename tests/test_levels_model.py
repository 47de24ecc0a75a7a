"""The level words of the one-CTA BFS in a CPU-thread model that runs the kernel's
turns (wgm_protocol.h): a thread that reads a level's flag late, with the first
thread already in the next level, must still find it raised."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("model") / "liblevels_model.so")
    subprocess.run(["g++", "-std=c++20", "-O2", "-fPIC", "-shared", "-pthread", "-o", out,
                    os.path.join(HERE, "model", "levels_model.cpp")], check=True)
    lib = C.CDLL(out)
    lib.model_levels.argtypes = [C.c_int, C.c_int, C.c_int, C.c_void_p]
    return lib


def _run(model, planted, threads, levels):
    out = np.zeros(2, np.int32)
    model.model_levels(planted, threads, levels, out.ctypes.data)
    return out.tolist()


@pytest.mark.parametrize("threads", [2, 5])
@pytest.mark.parametrize("levels", [1, 2, 3, 4, 50])
def test_a_late_reader_finds_its_level_s_flag(model, threads, levels):
    assert _run(model, 0, threads, levels) == [0, 0]


def test_planted_clear_of_the_flag_just_raised_is_caught(model):
    assert _run(model, 1, 3, 10)[0] > 0
