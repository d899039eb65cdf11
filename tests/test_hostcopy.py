"""Large copies between pageable host fields and the device (csrc/hostcopy.cuh) on
the CPU, against a fake of the CUDA runtime calls that it makes: whole at every
size, the caller's current device left alone, several threads and devices at
once, errors returned, the pinned set made when it pays and given back."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_hostcopy(tmp_path):
    exe = str(tmp_path / "hostcopy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-Wall", "-pthread", "-I",
                    os.path.join(HERE, "fake_cuda"), "-x", "c++",
                    os.path.join(HERE, "fake_cuda", "hostcopy_check.cc"), "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr
