"""CPU: kernel attributes and device addresses are kept for each device.  The
helper is checked with faked devices; the sources keep no such state in a
function-local static, which would hold what the first device returned."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "alamo_gb300", "csrc")


def test_state_is_kept_per_device(tmp_path):
    exe = str(tmp_path / "device_once_test")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-I", CSRC,
                           os.path.join(ROOT, "tests", "cpp", "device_once_test.cpp"), "-o", exe])
    assert subprocess.run([exe], timeout=60).returncode == 0


def test_no_device_state_in_a_static():
    calls = r"cudaFuncSetAttribute|cudaGetSymbolAddress|cudaDeviceGetAttribute|init_\w+_attributes"
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        src = re.sub(r"//[^\n]*", "", open(f).read())
        for m in re.finditer(r"\bstatic\s+(?:const\s+)?(?:bool|int)\s*\*?\s*\w+\s*=\s*[^;]*;", src):
            assert not re.search(calls, m.group(0)), (f, m.group(0))
