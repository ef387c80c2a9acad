"""CPU: the rule by which the resident kernels' CTAs wait for one another
(csrc/arrivals.cuh), over the wrap of its 32-bit count."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("arrivals") / "arrivals_wrap")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "gliomauq_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "arrivals_wrap.cpp"), "-o", out], check=True)
    return out


@pytest.mark.parametrize("ctas", [1, 2, 16, 152])
@pytest.mark.parametrize("start", ["0", "0xffffffff", "0xfffffff0", "0xfffff000", "0x7ffffffe"])
def test_no_barrier_is_passed_early_or_never(exe, ctas, start):
    p = subprocess.run([exe, str(ctas), start, "200", "7"], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout
