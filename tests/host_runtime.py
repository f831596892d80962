"""The library's host code on host_runtime.cpp: the package over a library linked from the built
objects and that runtime, in a process of its own, and the order of what it enqueued."""
from __future__ import annotations

import ctypes as C
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def build(folder) -> str:
    """The library over the host runtime (objects as build.py makes them); its path."""
    sys.path.insert(0, ROOT)
    import __graft_entry__ as entry

    recipe = entry._load_build_module()
    if not shutil.which("g++") or not (shutil.which("nvcc") or os.path.exists("/usr/local/cuda/bin/nvcc")):
        pytest.skip("needs g++ and the CUDA toolkit")
    recipe.build()
    objects = [os.path.join(recipe.BUILD, os.path.basename(s).replace(".cu", ".o")) for s in recipe.sources()]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(recipe.nvcc()))), "include")
    out = os.path.join(str(folder), "libs2d_host.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", include,
                    os.path.join(HERE, "host_runtime.cpp"), *objects, "-o", out, "-lpthread"], check=True)
    return out


def run(library: str, program: str) -> str:
    """`program` in a process of its own with `pkg` (the package over `library`) and `Record`."""
    head = (f"import sys; sys.path[:0] = [{ROOT!r}, {HERE!r}]\n"
            f"from host_runtime import *\npkg = load({library!r})\n")
    r = subprocess.run([sys.executable, "-c", head + program], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, f"exit {r.returncode}\n{r.stdout}\n{r.stderr}"
    return r.stdout


# ------------------------------------------------------------------ inside that process
def load(library: str):
    import __graft_entry__ as entry
    pkg = entry.load_package()
    host = C.CDLL(library)
    host.host_record.restype = C.c_char_p
    host.host_fail.argtypes = [C.c_char_p, C.c_int, C.c_int]
    host.host_capture.argtypes = [C.c_void_p, C.c_int]
    low = sys.modules[pkg.__name__ + "._lib"]
    low.LIB_PATH = library
    pkg.host = host
    return pkg


class Record:
    """The operations enqueued since host_forget(), with what each is ordered behind: the one
    before it on its stream, the operations of an event its stream waited for, and what the host
    had waited for by then."""

    def __init__(self, host):
        self.ops, self.before = [], []          # before[i]: bit set of the operations done before i
        done, host_done, recorded = {}, 0, {}
        for line in host.host_record().decode().splitlines():
            what, *rest = line.split()
            if what == "wait_event":
                host_done |= recorded.get(rest[0], 0)
                continue
            st = rest[0]
            if what == "wait_stream":
                host_done |= done.get(st, 0)
            elif what == "wait":
                done[st] = done.get(st, 0) | recorded.get(rest[1], 0)
            elif what == "record":
                recorded[rest[1]] = done.get(st, 0) | host_done
            elif what not in ("capture", "captured"):
                i = len(self.ops)
                self.ops.append((what, st, rest[1:]))
                self.before.append(done.get(st, 0) | host_done)
                done[st] = self.before[i] | (1 << i)

    def find(self, what, name=""):
        """Operations of a kind; kernels by a part of their name."""
        return [i for i, (w, _, rest) in enumerate(self.ops) if w == what and (not name or name in rest[0])]

    def ordered(self, a, b):
        return a == b or bool(self.before[max(a, b)] >> min(a, b) & 1)
