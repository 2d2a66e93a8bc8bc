"""The host thread pool. Runs on CPU."""
import os
import subprocess

import pytest

from msnhnet_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("pool") / "host_pool_check")
    subprocess.run([build._host_cxx(), "-O1", "-std=c++17", "-Wall", "-o", exe, os.path.join(HERE, "host_pool_check.cpp"), "-ldl", "-lpthread"], check=True)
    return exe


@pytest.mark.parametrize("may_start", [0, 1, 2, 6, 7, 100])
def test_jobs_are_done_however_few_threads_start(check, may_start):
    r = subprocess.run([check, str(may_start)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
