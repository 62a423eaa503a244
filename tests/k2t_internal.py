"""Functions of libkronos_cuda.so that are not part of the C interface, by their C++ names (namespace k2t)."""
import functools
import re
import subprocess

import kronos_2t_b200 as k2
from kronos_2t_b200 import ffi


@functools.lru_cache
def _symbols():
    return subprocess.run(["nm", "-D", "--defined-only", ffi.lib_path()], check=True, capture_output=True, text=True).stdout.split()


def internal(name, restype, *argtypes):
    found = [s for s in _symbols() if re.match(rf"_ZN3k2t{len(name)}{name}E", s)]
    assert len(found) == 1, (name, found)
    f = getattr(k2.load_library(), found[0])
    f.restype, f.argtypes = restype, list(argtypes)
    return f
