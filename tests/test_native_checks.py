"""Host-side rules of the device code, compiled and run on the CPU (tests/native)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mapol_b200", "csrc")


def run_native(tmp_path, name):
    """Compiles tests/native/<name>.cpp with the library's host sources; its output."""
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    exe = str(tmp_path / name)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I" + os.path.join(ROOT, "include"), "-I" + CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "native", name + ".cpp"), os.path.join(CSRC, "symbolic.cpp"),
                    os.path.join(CSRC, "synth.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    return out.stdout


def test_lane_pair_ranges_stay_inside_their_block(tmp_path):
    assert int(run_native(tmp_path, "lane_pairs_check").split()[1]) == 2 * 24 * (32 + 16 + 8)


def test_islands_without_supernodes_have_their_step_range(tmp_path):
    assert int(run_native(tmp_path, "island_plan_check").split()[1]) == 5 * 5 * 2


def test_plan_whose_upload_fails_is_built_again(tmp_path):
    assert run_native(tmp_path, "plan_cache_check").strip() == "ok"


def test_plans_are_refused_only_where_they_cannot_fit(tmp_path):
    out = run_native(tmp_path, "plan_needs_check").split()
    assert int(out[1]) > 100 and int(out[3]) > 30 and int(out[5]) > 40, out
