"""Host side of the kernel launches, over a fake CUDA runtime."""
import os
import subprocess

from godunov_mhd_ct_gb300.csrc import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_launch_leaves_no_error_behind(tmp_path):
    """A failed launch is reported by its return value only: as the thread's last error it would fail the next call of this
    library, or of any other in the process, that checks for one."""
    exe = str(tmp_path / "launch_error_check")
    cmd = [build.nvcc(), *build.ARCH, "-std=c++17", "-cudart", "none", os.path.join(HERE, "cpp", "launch_error_check.cu"),
           os.path.join(HERE, "cpp", "fake_cuda_runtime.cpp"), "-o", exe]
    subprocess.run(cmd, check=True, capture_output=True)
    reported, left, good, early = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert (reported, left, good, early) == (1, 0, 0, 1)
