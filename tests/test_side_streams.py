"""Side streams of the direct builds: nothing runs on them any more when a build
returns, also when it returns an error."""
import shutil
import subprocess
from pathlib import Path

import pytest

HOST = Path(__file__).resolve().parent / "host"
CSRC = HOST.parents[1] / "haskell-abinitio_gb300" / "csrc"


def test_a_scope_left_early_waits_for_the_side_streams(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "side_fork_check"
    subprocess.run([cxx, "-O1", "-std=c++17", "-Wall", "-Werror", "-I", str(HOST / "fake_cuda"), "-I", str(CSRC),
                    str(HOST / "side_fork_check.cpp"), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    runs = {}
    for line in out.splitlines():
        first, *calls = line.split("; ")
        name, status = first.split()
        runs[name] = (int(status), calls)
    fork = ["record 5 on 1", "wait 11 for 5", "wait 12 for 5", "wait 13 for 5"]
    join = [c for s, e in ((11, 21), (12, 22), (13, 23)) for c in (f"record {e} on {s}", f"wait 1 for {e}")]
    sync = ["sync 11", "sync 12", "sync 13"]
    assert runs["good"] == (0, fork + ["work"] + join)
    assert runs["error_in_work"] == (0, fork + ["work"] + sync)
    assert runs["not_forked"] == (0, [])
    assert runs["fails_1"] == (999, fork[:1])        # nothing was forked
    for at in range(2, 11):
        status, calls = runs[f"fails_{at}"]
        assert status == 999 and calls == (fork + join)[:at] + sync, at
