"""How interleaved regions are served: the host's rule and the length of a run, compiled from the header that the launcher uses."""
import ctypes
import os
import subprocess

import pytest

from tests.region_program import Load, Program, address, interleaved

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "functs_b200", "csrc")
EACH, AHEAD, WINDOW = 0, 1, 2
CODE = """
#include "region_plan.h"
extern "C" int program_size() { return sizeof(functs_b200_rprogram); }
extern "C" int plan(const functs_b200_rprogram* P, int rank, int inter, int* shared) {
    const fb::RegionPlan p = fb::region_plan(*P, rank, inter != 0);
    *shared = p.shared;
    return p.fetch;
}
extern "C" int words(int interleave, int elements, int base) { return fb::region_run_words(interleave, elements, base); }
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("region_plan")
    (d / "rule.cpp").write_text(CODE)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", str(d / "rule.so"), str(d / "rule.cpp")], check=True)
    lib = ctypes.CDLL(str(d / "rule.so"))
    assert lib.program_size() == ctypes.sizeof(Program)

    def plan(p, rank=1, inter=True):
        shared = ctypes.c_int(-1)
        fetch = lib.plan(ctypes.c_void_p(address(p)), rank, int(inter), ctypes.byref(shared))
        return fetch, shared.value
    plan.words = lib.words
    return plan


@pytest.mark.parametrize("width", range(2, 9))
def test_shared_memory_of_every_width(rule, width):
    """No form asks for more than six CTAs on an SM leave, let alone for more than a launch without opt-in may (48 KB)."""
    for loads in range(width + 1):
        fetch, shared = rule(interleaved(width, 606208, list(range(loads)), 1 << 20, 1 << 28))
        slots = width + loads
        if slots > 9 or loads == 0:
            assert fetch == (EACH if slots > 9 else AHEAD) and shared == 4096 * width
        elif width <= 4:
            assert fetch == WINDOW and shared == 2 * 4096 * width
        else:
            assert fetch == AHEAD and shared == 4096 * slots
        assert shared <= 36 * 1024


def test_what_one_run_cannot_serve(rule):
    def changed(fn):
        p = interleaved(3, 606208, [2, 1, 0], 1 << 20, 1 << 28)
        fn(p)
        return rule(p)[0]
    assert changed(lambda p: None) == WINDOW
    assert changed(lambda p: setattr(p.load[1], "tensor", 1)) == AHEAD
    assert changed(lambda p: setattr(p.load[1], "base", 3)) == AHEAD
    assert changed(lambda p: setattr(p.load[1], "base", -1)) == AHEAD
    assert changed(lambda p: p.load[2].coef.__setitem__(0, 6)) == AHEAD
    assert changed(lambda p: setattr(p.load[2], "dtype", 1)) == EACH
    p = interleaved(3, 606208, [2, 1, 0], 1 << 20, 1 << 28)
    assert rule(p, rank=2)[0] == AHEAD and rule(p, inter=False) == (EACH, 0)


def test_a_load_that_no_region_makes_does_not_stretch_the_run(rule):
    p = interleaved(4, 606208, [0, 1], 1 << 20, 1 << 28)
    assert rule(p)[0] == WINDOW
    p.load[p.num_loads] = Load(0, 0, 3, (ctypes.c_int32 * 4)(4))
    p.num_loads += 1
    assert rule(p)[0] == AHEAD


def test_a_run_ends_with_the_last_word_that_is_loaded(rule):
    for width in range(2, 9):
        for elements in (1, 2, 255, 1023, 1024):
            for bases in ([0], [width - 1], [width // 2, 0]):
                touched = {i * width + b for i in range(elements) for b in bases}
                assert rule.words(width, elements, max(bases)) == max(touched) + 1
