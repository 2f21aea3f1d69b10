"""The bitmap tier's scratch: sized for C candidates it holds every child of up
to C classes (no child is turned away on the device)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_arena_holds_every_child(tmp_path):
    exe = tmp_path / "arena_probe"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "gmbe_b200", "csrc"),
                    "-o", str(exe), os.path.join(ROOT, "tests", "probes", "arena_probe.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    for what, line in zip(("build", "run", "root"), out.splitlines(), strict=True):
        left, C, n, K = (int(x) for x in line.split())
        assert left >= 0, (what, left, C, n, K)
        print(what, left, C, n, K)
