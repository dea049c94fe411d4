"""The engine's book of device blocks (csrc/block_book.hpp), compiled for the host and
run on made-up addresses (tests/cpp/block_book.cpp): no device is involved."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("book") / "block_book")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-pthread", "-I",
                        os.path.join(ROOT, "gpu-preprocessor-ijoc_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "block_book.cpp"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("check", ["freed_elsewhere", "credit_returns"])
def test_book(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
