"""Downloads through the pinned staging when its allocation or one of its
launches fails (tests/stage_model.cpp, which replaces the library's pinned
allocation by one that can refuse)."""
from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

from code_mojo_gb300 import build

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def model(tmp_path_factory):
    lib = build.build_engine()
    exe = tmp_path_factory.mktemp("stage_model") / "stage_model"
    subprocess.run([build.NVCC, "-O1", "-std=c++17", "-I", str(ROOT / "include"), str(ROOT / "tests" / "stage_model.cpp"),
                    "-o", str(exe), "-L", str(lib.parent), "-lbfgpu", "-Xlinker", "--export-dynamic",
                    "-Xlinker", "-rpath", "-Xlinker", str(lib.parent)], check=True, capture_output=True)
    return exe


def run(model, what):
    r = subprocess.run([str(model), what], capture_output=True, text=True, env=dict(os.environ), timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_downloads_without_pinned_memory(model):
    run(model, "pinned")


def test_a_failed_download_leaves_nothing_in_flight(model):
    run(model, "drain")
