"""Compiles and runs a C++ program against the library's host-side headers."""
import os
import shutil
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "topopt_gb300", "csrc")


def run_cpp(tmp_path, source, *args):
    """The finished process of `source`, built as the library's host code is."""
    cc = shutil.which("g++") or shutil.which("c++")
    assert cc, "no C++ compiler"
    src, exe = tmp_path / "main.cpp", tmp_path / "main"
    src.write_text(source)
    built = subprocess.run([cc, "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-pthread",
                            "-I", CSRC, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    return subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=120)
