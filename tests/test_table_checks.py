"""tests/tables_check.cu: table loading with tables that no front end makes, on the CPU."""

import os
import resource
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    out = str(tmp_path_factory.mktemp("tables") / "tables_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-o", out,
                    os.path.join(HERE, "tables_check.cu")], check=True)
    return out


@pytest.mark.parametrize("case", ["arity", "sentinels", "productions"])
def test_tables_that_no_front_end_makes(exe, case):
    room = 4 << 30
    out = subprocess.run([exe, case], capture_output=True, text=True, timeout=120,
                         preexec_fn=lambda: resource.setrlimit(resource.RLIMIT_AS, (room, room)))
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.returncode, out.stderr)
