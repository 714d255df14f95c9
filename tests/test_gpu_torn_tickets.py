"""The counters that launches leave for the next one, as calls of one context
that overlapped would leave them (tests/cpp/torn_tickets.cu)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build(out_dir):
    lib = os.path.join(ROOT, "meshtrex_b200")
    exe = os.path.join(str(out_dir), "torn_tickets")
    cmd = ["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I",
           os.path.join(ROOT, "include"), "-I", os.path.join(lib, "csrc"),
           os.path.join(ROOT, "tests", "cpp", "torn_tickets.cu"), "-L", lib, "-lmeshtrex_b200", "-Xlinker",
           f"-rpath={lib}", "-o", exe]
    env = dict(os.environ, PATH=os.environ.get("PATH", "") + ":/usr/local/cuda/bin")
    r = subprocess.run(cmd, capture_output=True, text=True, env=env)
    assert r.returncode == 0, r.stderr
    return exe


def test_torn_ticket_program_builds(tmp_path):
    assert os.path.exists(_build(tmp_path))


@pytest.mark.gpu
def test_torn_tickets_are_reported_and_heal(tmp_path):
    r = subprocess.run([_build(tmp_path)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
