"""The split kernel's waiting lists hold every copy that its rounds can leave waiting."""

import pathlib
import subprocess

HERE = pathlib.Path(__file__).resolve().parent / "native"


def test_waiting_lists_are_long_enough_for_every_sequence_of_rounds(tmp_path):
    exe = tmp_path / "split_lists"
    subprocess.run(["g++", "-std=c++17", "-O2", str(HERE / "split_lists.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
