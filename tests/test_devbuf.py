"""Device buffers that share an allocation (csrc/devbuf.cu), on the CPU: tests/devbuf_check.cpp puts a counted
heap in place of cudaMalloc."""
import os
import subprocess

from minibude_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_growth_gives_back_what_it_outgrows(tmp_path):
    exe = str(tmp_path / "devbuf_check")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", B.CSRC, "-I", cuda, os.path.join(HERE, "devbuf_check.cpp"),
                        "-x", "c++", os.path.join(B.CSRC, "devbuf.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", (out.stdout, out.stderr)
