"""The network's device buffers over changing grids, on the CPU: a host
program (tests/cpp/net_buffers_check.cpp) runs csrc/net_buffers.h with a
counting allocator and compares what is held with what the kernels write."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_buffers_hold_what_the_kernels_write(tmp_path):
    exe = str(tmp_path / "net_buffers_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "liquidhairinteration_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "net_buffers_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.strip().endswith("ok: 0 failures"), r.stdout
