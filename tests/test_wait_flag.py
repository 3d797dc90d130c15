"""A wait of a tensor-core kernel that gives up is reported to the owner of the
launch, once, and to nobody else (csrc/host/wait_flag.h, compiled with the host
compiler; no GPU needed)."""
import json
import subprocess
from pathlib import Path


def test_expired_waits_are_reported_once_and_to_their_owner(tmp_path):
    src = Path(__file__).resolve().parent / "wait_flag_check.cpp"
    exe = tmp_path / "wait_flag_check"
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O2", "-pthread", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert r.returncode == 0 and out["mismatches"] == 0, out
