"""Device functions of the pooled kernels, compiled for the CPU as a warp of one lane."""

import pathlib
import subprocess

import pytest

from opengate_gb300 import build

HERE = pathlib.Path(__file__).resolve().parent / "native"


@pytest.fixture(scope="module")
def cuda_headers():
    return pathlib.Path(build.nvcc()).resolve().parents[1] / "include"


def _run(name, tmp_path, headers):
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", str(headers), str(HERE / f"{name}.cpp"),
                    "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True)


def test_walk_of_a_lane_without_a_slot_reads_no_table_out_of_range(tmp_path, cuda_headers):
    r = _run("walk_idle_lane", tmp_path, cuda_headers)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)


def test_launch_shapes(tmp_path, cuda_headers):
    r = _run("pool_shape", tmp_path, cuda_headers)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
