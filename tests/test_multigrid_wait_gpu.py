"""The multigrid solve's bounded waits: one that runs out is reported as an error status, once, and the solves
after it give what they gave before (native/multigrid_wait.cpp, built against the library)."""
import subprocess

import pytest

from rs_gb300 import build

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_reported_once(tmp_path):
    cuda = build._cuda_home()
    exe = tmp_path / "multigrid_wait"
    source = build.ROOT.parent / "tests" / "native" / "multigrid_wait.cpp"
    subprocess.run(
        [str(cuda / "bin" / "nvcc"), "-std=c++17", "-cudart", "shared", f"-I{build.INCLUDE}", f"-I{build.CSRC}", str(source),
         "-o", str(exe), str(build.LIB), "-Xlinker", f"-rpath={build.LIB.parent}"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.stdout, r.stderr)
