"""The cell arithmetic shared by host and device, on the CPU (compiled from the library's header)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_f64_cell_equals_the_reference_formula(tmp_path):
    import sph_build

    exe = str(tmp_path / "cell_axis")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "gmu-water-simulation_gb300", "csrc"), "-I",
                    os.path.join(sph_build._cuda_home(), "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "test_cell_axis.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, check=True)
    assert r.stdout.strip() == "0"
