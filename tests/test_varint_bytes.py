"""The varint decoder touches the coded bytes and nothing around them (the
buffer has no padding): its word reader compiled for the host under
AddressSanitizer, over every misalignment and up to four words."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "varint_bytes_main.cpp")
CSRC = os.path.join(ROOT, "distributed-string-sorting_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_reads_stay_inside(tmp_path):
    exe = str(tmp_path / "varint_bytes")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=address", "-I", CSRC, "-isystem",
                    os.path.join(CUDA, "include"), SRC, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, env=dict(os.environ, LD_PRELOAD=""))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr[-3000:]
