"""Host work over the cores (host_threads.h): a thread that cannot be started, for want of memory too, is done
without; the process never ends, and no item is lost."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    path = tmp_path_factory.mktemp("threads") / "check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", f"-I{os.path.join(ROOT, 'x3dcore2_gb300', 'csrc')}", "-o",
                    str(path), os.path.join(ROOT, "tests", "cpp", "host_threads_check.cpp")], check=True)
    return path


@pytest.mark.parametrize("n", [0, 1, 2, 64])
def test_allocations_that_fail(check, n):
    assert subprocess.run([str(check), str(n)], timeout=120).returncode == 0
