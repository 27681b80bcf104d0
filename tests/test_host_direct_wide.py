"""The direct defect solve's wide warp tiles and update sweep (bph_direct.h, the functions that the
kernel itself calls), emulated lane by lane on the CPU."""
import os
import subprocess

from tests.test_host_logic_cpp import CPP, CSRC


def test_wide_tiles_and_update_sweep(tmp_path):
    exe = tmp_path / "direct_wide_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC,
                    os.path.join(CPP, "direct_wide_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "all checks passed" in out.stdout
