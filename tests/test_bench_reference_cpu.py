"""bench.py --impl reference where the reference's own binary is missing: it says so and times nothing in its place. Runs on CPU."""
import json
import os
import shutil
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_without_the_binary_the_arm_is_unavailable(tmp_path):
    for name in ("bench.py", "msnhnet_b200", "oracle"):                   # the tree without oracle/_ref
        src = os.path.join(ROOT, name)
        if os.path.isdir(src):
            shutil.copytree(src, tmp_path / name, ignore=shutil.ignore_patterns("_ref", "_build", "__pycache__"))
        else:
            shutil.copy(src, tmp_path / name)
    r = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--gpus", "1", "--steps", "1", "--warmup", "1"], cwd=tmp_path,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["impl"] == "reference" and line["unavailable"] and "value" not in line
