"""The host threads that expand a packed pred (csrc/pred_expander.h), without a GPU: a C++ program stands in for the
kernel that marks the chunks and for the stream's state."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("pred_expander") / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "graph500_b200", "csrc"),
                    os.path.join(ROOT, "tests", "pred_expander_check.cc"), "-o", str(exe)], check=True,
                   env={k: v for k, v in os.environ.items() if k not in ("CC", "CXX")})
    return str(exe)


@pytest.mark.parametrize("check", ["entries", "unmarked", "refused_once", "does_not_fit", "long_wait", "few_threads"])
def test_expander(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "ok" and r.returncode == 0, (check, r.stdout, r.returncode)
