"""The gathered scale window of the z-marching conv on the CPU: the same header that the kernel includes, over every tile of small volumes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_gathered_window_bytes_and_bounds(tmp_path):
    """the window's bytes, and no load outside the scale plane: not even of the last word of a plane whose size is no multiple of four"""
    exe = str(tmp_path / "gather_window")
    subprocess.run([os.environ.get("CXX", "g++"), "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ufsm_b200", "csrc"), os.path.join(ROOT, "tests", "gather_window.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
