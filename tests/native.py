"""Runs a C++ snippet against the library's host code (no GPU): the body of a
main() that sees the headers of gpudock_b200/csrc and links libgpudock.so;
CHECK(x) ends it with the failing expression."""
import os
import shutil
import subprocess

from gpudock_b200 import build

CUDA = os.path.dirname(os.path.dirname(build.nvcc()))


def run(tmp_path, body, prelude=""):
    src, exe = str(tmp_path / "t.cc"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write('#include <cstdio>\n#include <cstdlib>\n#include "gd_common.h"\n'
                "#define CHECK(x) do { if (!(x)) { std::printf(\"line %d: %s\\n\", __LINE__, #x); "
                "std::exit(1); } } while (0)\n" + prelude + "\nint main() {\n" + body + "\n}\n")
    lib = build.build()
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", "-I", build.CSRC, "-I",
                    os.path.join(build.ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                    "-o", exe, src, lib, "-Wl,-rpath," + os.path.dirname(lib), "-pthread"],
                   check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    return res.stdout
