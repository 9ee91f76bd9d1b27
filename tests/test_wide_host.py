"""The roles of the persistent products and of the loader of portions' keys (tilemega_b200/csrc/wide.cuh) on host threads: tiles, stages and accumulators take their turns, and
whichever wait gives up, every role ends, behind the last product and copy."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_every_role_ends_whichever_wait_gives_up(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    binary = tmp_path / "wide_roles"
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-x", "c++", f"-I{ROOT / 'tilemega_b200' / 'csrc'}", str(ROOT / "tests" / "wide_roles.cpp"),
                    "-o", str(binary)], check=True)
    done = subprocess.run([str(binary)], capture_output=True, text=True, timeout=120)
    assert done.returncode == 0, done.stdout + done.stderr
