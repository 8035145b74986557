"""The places of a query's lists (tests/lists_unit.cpp), with totals past 31 and 32 bits."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_places_past_31_bits():
    with tempfile.TemporaryDirectory() as d:
        exe = os.path.join(d, "lists_unit")
        subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "box2d-rs_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "lists_unit.cpp"), "-o", exe], check=True)
        out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
