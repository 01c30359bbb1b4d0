"""Runs a script in a child process against the library linked with a CUDA
runtime that needs no device (fake_cuda.cpp): `ctx` is an open context, `native`
its module, `fake` the runtime."""
import os
import subprocess
import sys

import pytest

from ish_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))

PRELUDE = """
import ctypes as C
import re
import sys
import numpy as np
sys.path[:0] = [{root!r}, {here!r}]
from ish_gb300 import build, native
build.LIB = {lib!r}
fake = C.CDLL({lib!r})
fake.fake_report.restype = fake.fake_last_wave.restype = C.c_char_p
ctx = native.Context(0)
def last_wave():
    "(columns per thread, mode, layout, lean build) of the last wavefront kernel"
    return tuple(map(int, re.search(rb"_kernelILi(\\d+)ELi(\\d)ELi(\\d)ELi(\\d)E", fake.fake_last_wave()).groups()))
"""


def link(tmp) -> str:
    """The library over the fake runtime, linked into directory `tmp`."""
    build.build()
    objs = [os.path.join(build.BUILD, s[:-3] + ".o") for s in build.sources()]
    if not all(map(os.path.exists, objs)):
        build.build(force=True)
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    lib = os.path.join(tmp, "libish_fake.so")
    cmd = ["g++", "-std=c++17", "-O1", "-fPIC", "-fvisibility=hidden", "-shared", "-Wl,-Bsymbolic", "-I", cuda,
           os.path.join(HERE, "fake_cuda.cpp"), *objs, "-lpthread", "-o", lib]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lib


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    return link(str(tmp_path_factory.mktemp("fake")))


def run(lib, script):
    """The script's standard output; its failure is the test's."""
    code = PRELUDE.format(root=os.path.dirname(HERE), here=HERE, lib=lib) + script
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
