"""The batch autotuner's search, with made-up times in the place of runs."""

import pathlib
import subprocess

HERE = pathlib.Path(__file__).resolve().parent / "native"


def test_search_keeps_the_start_unless_a_point_is_faster(tmp_path):
    exe = tmp_path / "tune_search"
    subprocess.run(["g++", "-std=c++17", "-O1", str(HERE / "tune_search.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
