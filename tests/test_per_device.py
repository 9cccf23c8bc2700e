"""State that belongs to a device is kept per device: the holder (compiled for the host), and that
no kernel attribute or occupancy figure is kept once for the process."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "einsums_gb300", "csrc")


def test_holder(tmp_path):
    exe = str(tmp_path / "per_device_test")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", CSRC,
                    os.path.join(ROOT, "tests", "cpp", "per_device_test.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.strip() == "per device ok"


def test_no_device_state_of_the_process():
    """Statics that are initialised from calls on the current device, or under a once_flag."""
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"static (?!_)[^;{]*=\s*[^;]*;", text):
            assert not re.search(r"cudaFuncSetAttribute|cudaOccupancy|resident_grid", m.group(0)), (path, m.group(0))
        for m in re.finditer(r"call_once\((.*?)\n    \}\);", text, re.S):
            assert not re.search(r"cudaFuncSetAttribute|cudaOccupancy|attributes\(\)", m.group(1)), (path, m.group(1))
