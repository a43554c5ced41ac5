"""Two host threads that call the same routine with different sizes at the same time, each on its own stream: a
kernel's shared-memory limit belongs to the kernel, so the thread with the small launches must not lower it between
the other's opt-in and launch (that launch then fails and its output is not written)."""
import os
import subprocess

import pytest

from tests.helpers import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("threads") / "two_threads")
    lib, cuda = os.path.join(ROOT, "blasfeo_b200"), "/usr/local/cuda"
    subprocess.run(["gcc", "-O1", "-I" + os.path.join(ROOT, "include"), "-I" + cuda + "/include",
                    os.path.join(ROOT, "tests", "two_threads.c"), "-o", exe, "-L" + lib, "-lblasfeo_b200",
                    "-L" + cuda + "/lib64", "-lcudart", "-lpthread", "-Wl,-rpath," + lib + ":" + cuda + "/lib64"],
                   check=True)
    return exe


@pytest.mark.parametrize("op,n0,n1,calls", [("trsm", 64, 96, 20000), ("getrf", 132, 250, 8000), ("ric", 8, 16, 20000)])
def test_sizes_by_thread(program, op, n0, n1, calls):
    r = subprocess.run([program, op, str(n0), str(n1), str(calls)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, "failed calls of each thread: " + r.stdout + r.stderr
