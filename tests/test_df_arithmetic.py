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


def test_squares_have_no_bias(tmp_path):
    """Rounding averages out over the quartets that a G element sums, a bias does not.  A value's error is about
    2^-48 of it (32 units of 2^-53) at either sign, so the mean over 2 million values lies within 0.1 units of the bias.
    The square of the low float, left out, is one of 6 units; an unnormalised reciprocal square root's, of 40."""
    sq, rq = (float(v) for v in _run(tmp_path, "df_bias_main").split())
    assert abs(sq) < 0.25 and abs(rq) < 4.0, (sq, rq)
