"""The carry-chain arithmetic of the device header, compiled for the host,
against schoolbook sums on limbs that make carries run, and the quotients
it takes from double divisions."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_carry_chains_on_the_host(tmp_path):
    exe = str(tmp_path / "chaincheck")
    subprocess.run(["g++", "-std=c++17", "-O1", "-frounding-math", "-ffp-contract=off", "-o", exe, os.path.join(HERE, "devarith", "chaincheck.cpp")], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    lines = [ln.split() for ln in r.stdout.splitlines()]
    assert len(lines) >= 20 and all(int(ln[1]) > 0 and int(ln[2]) == 0 for ln in lines), r.stdout


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_products_by_halves_on_the_host(tmp_path):
    """The same with a limit of 24 limb pairs, so that short operands go by halves."""
    exe = str(tmp_path / "chaincheck")
    subprocess.run(["g++", "-std=c++17", "-O1", "-frounding-math", "-ffp-contract=off", "-DUP_MUL_UNROLL_PAIRS=24", "-o", exe,
                    os.path.join(HERE, "devarith", "chaincheck.cpp")], check=True)
    r = subprocess.run([exe, "60000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert sum(ln.startswith("mul<") for ln in r.stdout.splitlines()) >= 25
