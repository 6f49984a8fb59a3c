"""What follows from a bounded wait that ran out, on the host: no kernel runs and no wait runs out on a device."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "altopir-public_b200", "csrc")


@pytest.fixture(scope="module")
def waits(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("waits") / "waits")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, os.path.join(HERE, "cpp", "test_waits.cpp"), "-o", exe],
                   check=True)
    return lambda *args: subprocess.run([exe, *args], capture_output=True, text=True, timeout=300).stdout.strip()


def test_exchange_of_shares_after_a_lost_share(waits):
    assert waits() == "0"


def test_no_error_code_hides_another(waits):
    assert waits("codes") == "0"
