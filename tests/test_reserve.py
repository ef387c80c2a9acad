"""CPU: the allocations that stand or fall together (csrc/reserve.h), over an
allocator that fails. A set that is half there would be taken for the whole by
the next call, which writes through its null pointers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_buffer_or_none(tmp_path):
    exe = str(tmp_path / "reserve_fail")
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-I" + os.path.join(ROOT, "gliomauq_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "reserve_fail.cpp"), "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout
