"""The library's own objects linked with a CUDA runtime that has no device (fake_cudart.c), so that what the
host does with memory, copies, launches and graphs can be tested on the CPU: allocations that fail,
sizes that change, the launches a call makes."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


class FakeRuntime:
    """Control functions of fake_cudart.c."""

    def __init__(self, path):
        self.lib = C.CDLL(path)
        for name, args, res in (("room", [C.c_size_t], None), ("used", [], C.c_size_t), ("peak", [], C.c_size_t), ("refuse", [C.c_long], None),
                                ("refuse_graphs", [C.c_int], None), ("refuse_downloads", [C.c_int], None),
                                ("blocks_per_sm", [C.c_int], None), ("violations", [], C.c_long),
                                ("instantiations", [], C.c_long), ("launches", [], C.c_long), ("mallocs", [], C.c_long),
                                ("watch", [C.c_char_p, C.c_char_p], C.c_int), ("log", [], C.c_long),
                                ("log_watch", [C.c_long], C.c_int), ("log_grid", [C.c_long], C.c_uint),
                                ("log_arg", [C.c_long, C.c_int], C.c_longlong),
                                ("log_room", [C.c_long, C.c_int], C.c_longlong), ("reset", [], None), ("clear_watches", [], None)):
            fn = getattr(self.lib, "fake_" + name)
            fn.argtypes, fn.restype = args, res
            setattr(self, name if name not in ("watch", "log") else "_" + name, fn)
        self._names = {}

    def watch(self, part, sig):
        self._names[self._watch(part.encode(), sig.encode())] = (part, sig)

    def launches_of(self, part):
        """The logged launches of one watched kernel: grid, argument values, and for each pointer the bytes that
        its block had from there on at the launch."""
        out = []
        for k in range(self._log()):
            name, sig = self._names[self.log_watch(k)]
            if name == part:
                out.append((self.log_grid(k), [self.log_arg(k, i) for i in range(len(sig))],
                            [self.log_room(k, i) for i in range(len(sig))]))
        return out


def link(tmp):
    if shutil.which("gcc") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime_api.h")):
        pytest.skip("gcc or the CUDA headers are not installed")
    import importlib
    importlib.import_module("phlegethon_b200.build").build(force=False)
    objs = [os.path.join(ROOT, "phlegethon_b200", "_build", o) for o in ("phl_runtime.o", "phl_split.o")]
    fake, out = os.path.join(str(tmp), "fake.o"), os.path.join(str(tmp), "libphl_host.so")
    subprocess.run(["gcc", "-O1", "-fPIC", "-I", os.path.join(CUDA, "include"), "-c",
                    os.path.join(ROOT, "tests", "fake_cudart.c"), "-o", fake], check=True)
    # -Bsymbolic: the library's calls stay with this runtime even where a real one is loaded too
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", out, *objs, fake], check=True)
    return out
