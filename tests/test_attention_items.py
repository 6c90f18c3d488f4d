"""The host-compilable part of the attention kernel's index arithmetic, compiled and walked on the CPU."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_unit_once_and_no_address_outside(tmp_path):
    program = tmp_path / "check"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT.parent / 'bionemo_inference_runtime_b200/csrc'}",
                    str(ROOT / "attention_items_check.cpp"), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True)
    assert done.returncode == 0 and done.stdout == "ok\n", done.stdout
