"""The host threads of uploads and downloads hand every error to the caller
(CPU; tests/native/host_runs_check.cpp, built with g++), and the transfers use
nothing else to start threads."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "culs_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_errors_of_every_run_reach_the_caller(tmp_path):
    exe = tmp_path / "host_runs_check"
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-pthread", "-I", str(CSRC),
                           str(ROOT / "tests" / "native" / "host_runs_check.cpp"), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "bad 0" in out.stdout


@pytest.mark.parametrize("name", ["aiger_dev.cu", "host_io.cu"])
def test_transfers_drop_no_copy_error(name):
    """Every copy's result is used (assigned, tested or returned), and threads
    start through run_parallel alone."""
    text = (CSRC / name).read_text()
    assert "std::thread" not in text and "run_parallel" in text
    upload = text[text.index("int Engine::upload"):]
    upload = upload[:upload.index("\n}\n")]
    assert re.findall(r"cudaMemcpyAsync", upload)
    assert not re.findall(r"^\s*cudaMemcpyAsync", upload, re.M)
