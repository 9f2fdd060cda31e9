"""CPU tests of csrc/host_rules.h, compiled with the host compiler."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"


def test_host_rules(tmp_path):
    exe = str(tmp_path / "host_rules_demo")
    r = subprocess.run([CXX, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I",
                        os.path.join(ROOT, "dda_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "host_rules_demo.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
