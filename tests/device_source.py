"""Compiles a C++ program against the library's device code as host code."""
import os
import re
import subprocess

from conftest import REPO

CSRC = os.path.join(REPO, "pcr_b200", "csrc")


def run(tmp_path, program: str) -> str:
    """Builds tests/cpp/`program` with device.cuh and returns its output."""
    with open(os.path.join(CSRC, "device.cuh")) as f:
        text = f.read()
    text, n = re.subn(r'asm\("rcp\.approx.*?;\\?.*?\);', "r = some_reciprocal(x);", text)
    text, m = re.subn(r'asm\("sqrt\.approx.*?;\\?.*?\);', "r = std::sqrt(x);", text)
    assert n == 1 and m == 1
    text = re.sub(r"#pragma unroll.*", "", text)
    (tmp_path / "device_host.h").write_text(text)
    exe = str(tmp_path / "program")
    subprocess.run(["g++", "-O2", "-w", "-std=c++17", "-mfma", "-ffp-contract=fast", "-I", str(tmp_path), "-I", CSRC,
                    "-I", os.path.join(REPO, "include"), "-I", os.path.join(REPO, "tests", "cpp"),
                    "-I", "/usr/local/cuda/include", "-o", exe, os.path.join(REPO, "tests", "cpp", program)], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout
