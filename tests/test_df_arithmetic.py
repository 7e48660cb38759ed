"""The arithmetic of the pairs of floats (df64.cuh, df_roots.cuh) run on the host, with the CUDA intrinsics it is
made of replaced by their IEEE meaning."""
import os
import subprocess

from conftest import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, name):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I" + os.path.join(CUDA, "include"),
                    "-I" + os.path.join(ROOT, "unomol_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", name + ".cpp"),
                    "-o", exe], check=True)
    return subprocess.run([exe], check=True, capture_output=True, text=True).stdout


def test_root_tables_are_read_inside_their_blocks(tmp_path):
    """Every T, whatever its split into two floats, takes the interval it lies in, up to the last of its table:
    an interval past the end holds NaN here (on the device, another block's numbers)."""
    out = _run(tmp_path, "df_roots_main")
    looked, wrong = (int(v) for v in out.strip().split("\n")[-1].split())
    assert looked > 1_000_000 and wrong == 0, out


def test_squares_of_differences(tmp_path):
    """(P - Q)^2 of close product centres: nothing of the size of an ulp of the coordinates, squared, is lost."""
    looked, wrong = (int(v) for v in _run(tmp_path, "df_diff_main").split())
    assert looked == 320_000 and wrong == 0, wrong
