"""A bounded wait that a kernel gives up is reported: by every later call on the context, by replays and by
the synchronising calls (native/wait_report.cu sets the flag from the host); and the kernel that gave it up ends
in order (native/wait_limit.cu lets every wait run out)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


def build_native(name, out_dir):
    """tests/native/<name>.cu against the library and its internal headers."""
    lib = os.path.join(ROOT, "shmoai_b200", "_build")
    exe = os.path.join(str(out_dir), name)
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                    os.path.join(ROOT, "tests", "native", name + ".cu"), "-L" + lib, "-lshmoai_b200",
                    "-Xlinker", "-rpath," + lib, "-o", exe], check=True)
    return exe


@pytest.mark.gpu
def test_given_up_wait_is_reported(tmp_path):
    r = subprocess.run([build_native("wait_report", tmp_path)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("args,tma", [
    (("conv",), "1"),
    (("ctpt", "100"), "1"), (("ctpt", "768"), "1"),  # X tiles ahead; one resident tile
    (("ctpt", "100"), "0"), (("ctpt", "768"), "0"),  # operands copied by the producer warps
    (("ctpt", "1000"), "1")])                        # a tile per CTA
def test_given_up_wait_ends_in_order(tmp_path, args, tma):
    r = subprocess.run([build_native("wait_limit", tmp_path), *args], capture_output=True, text=True, timeout=300,
                       env={**os.environ, "SHMOAI_CTPT_TMA": tma})
    assert r.returncode == 0, r.stdout + r.stderr
