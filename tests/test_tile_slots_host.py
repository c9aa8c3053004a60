"""The slots of the shared-memory Gram (doublyexcited_b200/csrc/tile_slots.h, the
code gram_tile.cu runs) over every shape the dispatch can pass, compiled for the
host: never past the tables, refused exactly where the distinct columns or two
stages do not fit."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "doublyexcited_b200", "csrc")


def test_slots_of_every_shape(tmp_path):
    exe = str(tmp_path / "tile_slots_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-fsanitize=undefined", "-I", CSRC,
                    os.path.join(HERE, "tile_slots_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and not r.stderr, r.stdout[-2000:] + r.stderr[-2000:]
