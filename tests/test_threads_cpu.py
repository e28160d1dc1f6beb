"""The host's parallel loop and its set-up once per device
(dmft-ed-zt_b200/csrc/host_threads.h), built into tests/threads_check.cpp with
the host compiler: every index once, the function's exception reaches the
caller, and where no thread can be made the calling one does the work instead of
the process ending; no thread passes set-up that another has only begun."""

import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_host_threads(tmp_path):
    exe = str(tmp_path / "threads_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(PKG_DIR, "csrc"),
                    os.path.join(ROOT, "tests", "threads_check.cpp"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stdout, r.stderr)
