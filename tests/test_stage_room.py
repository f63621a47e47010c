"""The staging room of a call's uploads is not refilled while a copy may still read it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_room_is_not_refilled_under_a_late_copy(tmp_path):
    out = str(tmp_path / "stage_room")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-I", os.path.join(ROOT, "bernasconi-krylov_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_stage_room.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

