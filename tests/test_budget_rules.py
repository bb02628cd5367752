"""Register budgets of the thread-per-link kernels by lattice size (budget.h,
host rules): which lattices take which, and what a mapping tuned on one lattice
does to lattices of another size."""
import ctypes
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "askja_b200", "csrc")


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("budget")
    src = d / "b.cpp"
    src.write_text('#include "budget.h"\nextern "C" {\n'
                   "int ahead(int N, long V) { return askja::force_ahead(N, V); }\n"
                   "int untuned(int N, int fp64, int residual, long V) {\n"
                   "  return askja::default_occupancy(N, fp64, residual, V); }\n"
                   "int carried(int t, int path, int N, int fp64, int residual, long V0, long V) {\n"
                   "  return askja::carried_occupancy(t, path, N, fp64, residual, V0, V); }\n}\n")
    so = d / "b.so"
    subprocess.check_call(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(so)])
    L = ctypes.CDLL(str(so))
    L.ahead.argtypes = [ctypes.c_int, ctypes.c_long]
    L.untuned.argtypes = [ctypes.c_int] * 3 + [ctypes.c_long]
    L.carried.argtypes = [ctypes.c_int] * 5 + [ctypes.c_long] * 2
    return L


def test_untuned_budgets(rules):
    one_wave, big = 2 * 148 * 32, 2048 * 32
    for V, ahead, fp64_su2 in ((1, 1, 0), (one_wave, 1, 0), (one_wave + 1, 0, 2), (big, 0, 2), (big + 1, 0, 0)):
        assert rules.ahead(2, V) == rules.ahead(3, V) == ahead and rules.ahead(4, V) == 0
        assert rules.untuned(2, 1, 0, V) == fp64_su2
        assert rules.untuned(3, 1, 0, V) == rules.untuned(4, 1, 0, V) == 0
    for N, small, large in ((2, 0, 2), (3, 0, 2), (4, 0, 0)):
        assert rules.untuned(N, 0, 1, 4 * 148 * 32) == small
        assert rules.untuned(N, 0, 1, 4 * 148 * 32 + 1) == large
        assert rules.untuned(N, 0, 0, 10**6) == 0  # without residual planes


@pytest.mark.parametrize("N,fp64,residual", [(2, 0, 1), (3, 0, 1), (4, 0, 1), (2, 1, 0), (3, 1, 0), (4, 1, 0), (3, 0, 0)])
def test_a_tuned_budget_stays_with_lattices_of_its_kind(rules, N, fp64, residual):
    sizes = (16, 8**4, 2 * 148 * 32, 2 * 148 * 32 + 1, 4 * 148 * 32 + 1, 16**4, 24**4, 32**4)

    def kind(V):
        return rules.untuned(N, fp64, residual, V), fp64 and rules.ahead(N, V)

    for V0 in sizes:
        for V in sizes:
            for tuned in (0, 1, 2):
                got = rules.carried(tuned, 0, N, fp64, residual, V0, V)
                assert got == (tuned if kind(V) == kind(V0) else rules.untuned(N, fp64, residual, V)), (V0, V, tuned)
                # the row kernels' budget does not depend on the lattice
                assert rules.carried(tuned, 1, N, fp64, residual, V0, V) == tuned
    # FP32 SU(3): tuned on 8^4, used on 32^4, and the reverse
    assert rules.carried(0, 0, 3, 0, 1, 8**4, 32**4) == 2 and rules.carried(2, 0, 3, 0, 1, 32**4, 8**4) == 0
