"""The launch rules' multiprocessor count is the current device's, and no literal."""
import os
import re
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "hemelb_gb300", "csrc")


def test_count_of_the_current_device(tmp_path):
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(os.environ.get("NVCC", "nvcc")))))
    exe = tmp_path / "sm_count"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", SRC, "-I", os.path.join(cuda, "include"),
                    os.path.join(ROOT, "tests", "cpp", "sm_count.cc"), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_literal_count_in_the_launch_code():
    for name in sorted(os.listdir(SRC)):
        with open(os.path.join(SRC, name)) as f:
            code = re.sub(r"//[^\n]*", "", f.read())
        found = re.findall(r"(?<![\w.])(?:152|304|1216|1215)(?![\w.])[^\n]*", code)
        assert name == "sm_count.h" or not found, (name, found)
