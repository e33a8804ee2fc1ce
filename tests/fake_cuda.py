"""The package on a stand-in for the CUDA runtime (tests/cpp/fake_cudart.cpp):
its objects linked with one that keeps device memory on the host, notes the
launches without running them, and fails where it is told to."""
from __future__ import annotations

import ctypes as C
import importlib.util
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "nbody-sim_b200")
OBJECTS = os.path.join(PACKAGE, "_build")


def load(folder):
    """(package, fake): a second instance of the package, on the stand-in; None
    where the library's objects have not been built."""
    objs = sorted(os.path.join(OBJECTS, f) for f in os.listdir(os.path.join(PACKAGE, "csrc"))
                  if f.endswith((".cu", ".cpp")))
    objs = [o + ".o" for o in objs]
    if not all(map(os.path.exists, objs)):
        return None
    path = os.path.join(str(folder), "libfake.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-o", path,
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp"), *objs], check=True)
    spec = importlib.util.spec_from_file_location("nbody_on_a_fake",
                                                  os.path.join(PACKAGE, "__init__.py"))
    nb = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = nb  # its dataclasses look themselves up
    spec.loader.exec_module(nb)
    nb.LIB_PATH = path
    nb.lib = nb._load()
    fake = C.CDLL(path)
    fake.fake_fail_launch.argtypes = [C.c_char_p, C.c_long]
    fake.fake_fail_alloc.argtypes = [C.c_long]
    fake.fake_names.restype = C.c_char_p
    fake.fake_launches.restype = fake.fake_bad_frees.restype = C.c_long
    fake.fake_pointer.argtypes, fake.fake_pointer.restype = [C.c_char_p, C.c_int], C.c_void_p
    return nb, fake
