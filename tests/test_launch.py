"""Host-side choices about launches (tests/launch_unit.cpp), and that what belongs to a device is kept for each
device: no function attribute or occupancy behind a flag of the whole process."""
import glob
import os
import re
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "box2d-rs_gb300", "csrc")


def test_choices():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "launch_unit")
        subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, os.path.join(ROOT, "tests", "launch_unit.cpp"),
                        "-o", exe], check=True)
        out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_what_belongs_to_a_device_is_kept_for_each():
    flag = re.compile(r"^\s+static (?:const )?(?:bool|int|cudaError_t) \w+ *=", re.M)
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = open(path).read()
        assert not flag.search(src), (os.path.basename(path), flag.search(src).group())
