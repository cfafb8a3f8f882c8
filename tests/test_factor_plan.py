"""The host side of the sparse factorisation on the CPU: tests/factor_plan_host.cpp, linked against the library."""
import os
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
