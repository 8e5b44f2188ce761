"""The operand rings of the tcgen05 kernels on the host: whichever bounded wait gives up, every copy that was
issued is waited for before the kernel's order returns (csrc/bpx_ring.h)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rings_leave_no_copy_in_flight(tmp_path):
    exe = str(tmp_path / "ring_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I" + os.path.join(ROOT, "fdt_b200", "csrc"),
                    os.path.join(ROOT, "tests", "c_host", "ring_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
