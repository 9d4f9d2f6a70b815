"""CPU: the bookkeeping of status words in flight (csrc/status_board.h) against a model of streams and events."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("status_board") / "model")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O1", "-pthread",
                    "-I" + os.path.join(ROOT, "hdla_impl_b200", "csrc"),
                    os.path.join(ROOT, "tests", "model", "status_board_model.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("what", ["lagging", "owner", "bounded", "reports"])
def test_status_board(model, what):
    r = subprocess.run([model, what], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
