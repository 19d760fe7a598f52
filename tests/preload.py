"""Functions of libdgcu replaced for one child process: a C++ source that
defines some of the library's internal functions (same namespace and
signature, from its headers), loaded ahead of it."""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "hopefoam_gb300", "csrc")


def compile_host(src, out, *more):
    """`src` (text) and the files in `more` as a shared library of host code."""
    cpp = str(out) + ".cpp"
    with open(cpp, "w") as f:
        f.write(src)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                        "-I", "/usr/local/cuda/include", cpp, *more, "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(out)


def run(so, code, *args, timeout=300):
    """`code` in a child process with `so` loaded first; its output."""
    before = lambda *p: ":".join(filter(None, p))
    env = dict(os.environ, LD_PRELOAD=before(so, os.environ.get("LD_PRELOAD")),
               PYTHONPATH=before(ROOT, HERE, os.environ.get("PYTHONPATH")))
    r = subprocess.run([sys.executable, "-c", code, *map(str, args)], cwd=ROOT, env=env, capture_output=True, text=True,
                       timeout=timeout)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
