"""CPU: the library thread that answers the MSM's last step (msm_answer.hpp,
compiled for the host), with the driver msm_answer_check.cpp in the kernel's
place."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CASES = ["no thread to be had", "ready long after", "kernel not launched", "many at once", "one core for both",
         "exit while watched"]


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = tmp_path_factory.mktemp("msm_answer") / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-o", str(exe),
                    os.path.join(HERE, "msm_answer_check.cpp"), "-ldl"], check=True)
    return str(exe)


@pytest.mark.parametrize("case", CASES)
def test_answering_thread(driver, case):
    subprocess.run([driver, case], check=True, timeout=60)
