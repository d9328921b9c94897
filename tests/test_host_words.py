"""The pinned words that kernels publish lengths in (HostWords, csrc/b2m_context.h)
are not given to another call, and not freed, while a kernel still has to write
them. host_words_check.cpp runs the class against a fake of the CUDA runtime;
no GPU is needed."""
import os
import subprocess

import b200mul

TESTS = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.dirname(b200mul.LIB_PATH)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_words_outlive_the_publications_they_are_owed(tmp_path):
    exe = str(tmp_path / "host_words_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(os.path.dirname(PKG), "include"), "-I", os.path.join(CUDA, "include"),
                    os.path.join(TESTS, "host_words_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
