"""The queue in which a warp of the direct builds collects the kets that pass the
screening, run on the host by 32 threads under the address and thread checkers."""
import shutil
import subprocess
from pathlib import Path

import pytest

HOST = Path(__file__).resolve().parent / "host"
CSRC = HOST.parents[1] / "haskell-abinitio_gb300" / "csrc"


@pytest.mark.parametrize("sanitizer", ["address,undefined", "thread"])
def test_every_survivor_once_and_in_range(tmp_path, sanitizer):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "queue_check"
    cmd = [cxx, "-O1", "-std=c++20", "-pthread", "-I", str(CSRC), str(HOST / "queue_check.cpp"), "-o", str(exe)]
    checked = subprocess.run(cmd + [f"-fsanitize={sanitizer}"], capture_output=True, text=True)
    if checked.returncode != 0:   # no sanitizer library here
        subprocess.run(cmd, check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    rows = [line.split() for line in r.stdout.splitlines()]
    for pattern, tasks, want, once, faults in rows[:4]:
        assert int(tasks) > 70 and int(want) > 70 and once == want and faults == "0", pattern
    assert rows[4] == ["in", "1005", "1", "0"] and rows[5] == ["out", "1000", "0", "1"]
