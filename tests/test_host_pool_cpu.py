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


QUOTAS = [("0::/\n", {"cpu.max": "max 100000"}, 0),
          ("0::/\n", {"cpu.max": "200000 100000"}, 2),
          ("0::/a/b\n", {"a/cpu.max": "250000 100000", "a/b/cpu.max": "max 100000"}, 3),             # an ancestor's limit, rounded up
          ("0::/a/b\n", {"a/cpu.max": "800000 100000", "a/b/cpu.max": "150000 50000"}, 3),
          ("0::/a\n", {}, 0),                                                                       # no such files
          ("3:cpuset:/x\n2:cpu,cpuacct:/docker/1\n", {"cpu,cpuacct/docker/1/cpu.cfs_quota_us": "400000", "cpu,cpuacct/docker/1/cpu.cfs_period_us": "100000"}, 4),
          ("1:cpu:/\n0::/\n", {"cpu/cpu.cfs_quota_us": "-1", "cpu/cpu.cfs_period_us": "100000"}, 0),
          ("1:cpu:/j\n0::/k\n", {"cpu/j/cpu.cfs_quota_us": "50000", "cpu/j/cpu.cfs_period_us": "100000", "k/cpu.max": "300000 100000"}, 1),
          ("4:cpuset:/s\n", {"cpuset/s/cpu.cfs_quota_us": "100000", "cpuset/s/cpu.cfs_period_us": "100000"}, 0)]   # not the cpu controller


@pytest.mark.parametrize("groups,files,want", QUOTAS)
def test_quota_of_the_control_groups(check, tmp_path, groups, files, want):
    (tmp_path / "groups").write_text(groups)
    for name, text in files.items():
        path = tmp_path / "root" / name
        path.parent.mkdir(parents=True, exist_ok=True)
        path.write_text(text + "\n")
    r = subprocess.run([check, "quota", str(tmp_path / "groups"), str(tmp_path / "root")], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and int(r.stdout) == want, r.stdout + r.stderr


@pytest.mark.parametrize("cpus,quota,want", [(16, 0, 7), (224, 0, 7), (224, 2, 1), (224, 1, 0), (224, 64, 7), (8, 0, 3), (8, 6, 3), (2, 0, 0), (1, 0, 0)])
def test_threads_stay_within_the_quota(check, cpus, quota, want):
    r = subprocess.run([check, "workers", str(cpus), str(quota)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and int(r.stdout) == want, r.stdout + r.stderr
