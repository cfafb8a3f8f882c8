"""The host side of the sparse factorisation on the CPU: tests/factor_plan_host.cpp, linked against the library."""
import os
import resource
import subprocess

import pytest

from tissueorigami_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("factor_plan") / "factor_plan_host")
    lib_dir = os.path.dirname(build.build())
    cuda = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "tissueorigami_b200", "csrc"),
           "-isystem", cuda, os.path.join(HERE, "factor_plan_host.cpp"), "-L", lib_dir, "-ltf_b200",
           f"-Wl,-rpath,{lib_dir}", "-pthread", "-o", exe]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr

    def run(*args, **kw):
        res = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, **kw)
        assert res.returncode == 0, f"{res.returncode} {res.stdout} {res.stderr}"
        return res.stdout.split()

    return run


@pytest.mark.parametrize("k", [0, 238609294, 238609295, 2**31 - 2])
def test_offsets_of_jacobian_values_do_not_wrap(host, k):
    """Nine doubles a block: from block 2^31 / 9 on their offsets need more than 32 bits."""
    assert host("span", k, k + 1) == [str(9 * k), str(9 * (k + 1))]


@pytest.mark.parametrize("limit", [1e8, 3e9, 3e11])
@pytest.mark.parametrize("nx,ny", [(500, 250), (2000, 50)])
def test_dissection_ends_where_the_limit_is_passed(host, nx, ny, limit):
    """A tissue whose factorisation is too large is not dissected to the end: the operations counted by then exceed
    the limit by no more than the root front's 2/3 p^3 (the largest front of such a sheet without boundary) and
    the fronts of a depth below it (as much again, with their boundaries ten times)."""
    ok, flops, _, fronts, _ = host("plan", nx, ny, 4, limit, 0, 1)
    whole = float(host("plan", nx, ny, 4, 1e15, 0, 1)[1])
    assert whole > 3e9
    if whole <= limit:
        assert ok == "1"
        return
    root = 2.0 / 3.0 * (12 * min(nx, ny)) ** 3
    assert (ok, fronts) == ("0", "0") and limit < float(flops) <= limit + 10 * root and float(flops) < whole


@pytest.mark.parametrize("sheet", [(1, 1, 1, 0), (3, 2, 2, 0), (31, 23, 4, 0), (40, 35, 3, 0), (40, 35, 1, 2), (60, 50, 2, 7),
                                   (9, 300, 1, 1)])
def test_boundaries_of_the_fronts(host, sheet):
    """Every column a pivot of one front; every front's boundary what its subtree touches, also around a column
    with hundreds of neighbours (found from the other side there)."""
    assert host("check", *sheet) == ["1", "0"]


def _limited(what, value):
    return lambda: resource.setrlimit(what, (value, resource.getrlimit(what)[1]))


def test_plan_without_threads(host):
    """Where no thread can be started (here: no address space for a stack of 64 TB), the caller's does it all."""
    args = ("plan", 60, 50, 2, 3e11, 0, 3)
    alone = host(*args, preexec_fn=_limited(resource.RLIMIT_STACK, 1 << 46))
    with_threads = host(*args)
    assert alone[0] == "1" and alone[:2] + alone[3:] == with_threads[:2] + with_threads[3:]


def test_plan_without_host_memory(host):
    """Too little memory, at whatever point of the plan: an exception for the caller, not the end of the process."""
    ways = [host("plan", 150, 100, 3, 1e15, 1, 3, kb)[0] for kb in [100 * 2**k for k in range(14)]]
    assert set(ways) == {"bad_alloc", "1"}


@pytest.mark.parametrize("every", [1, 7, 1000])
def test_no_plan_for_positions_that_are_not_numbers(host, every):
    """They cannot be ordered for the cuts; the iterative solve reports what becomes of such a tissue."""
    assert host("nan", 100, 100, every) == ["0"]
