"""pages_present (csrc/host_pages.h): a readout into arrays whose pages are there starts no
threads to make them present."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pages_of_host_arrays(tmp_path):
    exe = tmp_path / "host_pages"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "hemelb_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "host_pages.cc"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
