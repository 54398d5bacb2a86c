"""Function attributes and SM counts belong to a device, not to the process: the
set-up of csrc/per_device.h on the host, and no kernel set up for the process."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bem2d_gb300", "csrc")


def test_once_per_device(tmp_path):
    exe = str(tmp_path / "per_device")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", "per_device_host.cpp")], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout == "ok\n"


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC)
                                        if f.endswith((".cu", ".cuh"))))
def test_nothing_is_set_up_once_per_process(name):
    """No process-wide flag or initialiser around an attribute or device property."""
    text = open(os.path.join(CSRC, name)).read()
    assert "once_flag" not in text
    for m in re.finditer(r"static (?:const )?(?:int|bool|cudaError_t) \w+ =[^;]*?cuda\w+", text):
        assert False, m.group(0)
