"""The engine linked with tests/fake_cudart.cpp: its host code on a CPU, every
stream operation recorded, for tests of ordering, capture and allocation."""
from __future__ import annotations

import ctypes
import glob
import importlib.util
import json
import os
import subprocess
import sys
from dataclasses import dataclass

from cm_decrypt__b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
GLOBAL_CAPTURE, THREAD_LOCAL_CAPTURE = 0, 1


@dataclass(frozen=True)
class Op:
    call: int
    stream: int
    index: int
    name: str
    dst: int
    bytes: int
    arg: tuple
    seen: dict

    def after(self, other: "Op") -> bool:
        """Whether `other` has ended before this starts, on any timing."""
        return self.seen.get(other.stream, 0) >= other.index

    def writes(self, other: "Op") -> bool:
        """Whether this copy or memset overlaps the other's destination."""
        return self.bytes and other.bytes and self.dst < other.dst + other.bytes and other.dst < self.dst + self.bytes


class Fake:
    """cmd: the package over the linked library; rt: the runtime's own calls."""

    def __init__(self, tmp: str):
        build.build()
        obj, so, script = (os.path.join(tmp, f) for f in ("fake_cudart.o", "libcmd_fake.so", "exports"))
        include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))), "include")
        subprocess.run(["g++", "-std=c++20", "-O1", "-fPIC", "-I", include, "-c",
                        os.path.join(HERE, "fake_cudart.cpp"), "-o", obj], check=True)
        with open(script, "w") as f:  # nothing else: the real library may be in the same process
            f.write("{ global: cmd_*; fake_*; cuda*; local: *; };\n")
        objs = [o for o in glob.glob(os.path.join(build.BUILD, "*.o")) if not o.endswith("cli.cpp.o")]
        subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", f"-Wl,--version-script={script}", "-o", so, *sorted(objs),
                        obj, "-lpthread"], check=True)
        spec = importlib.util.spec_from_file_location("cmd_fake", os.path.join(build.PKG, "__init__.py"))
        self.cmd = importlib.util.module_from_spec(spec)
        sys.modules["cmd_fake"] = self.cmd
        spec.loader.exec_module(self.cmd)
        self.cmd.LIB_PATH = so
        self.cmd.lib()
        self.rt = ctypes.CDLL(so)
        self.rt.fake_ops.restype = ctypes.c_char_p
        self.rt.fake_allocated.restype = ctypes.c_size_t
        self.rt.fake_largest_malloc.argtypes = [ctypes.c_size_t]
        self.rt.fake_total.argtypes = [ctypes.c_size_t]
        self.rt.fake_elapsed.argtypes = [ctypes.c_float]
        self.reset()

    def reset(self):
        self.rt.fake_largest_malloc(2 ** 63)
        self.rt.fake_total(2 ** 63)
        self.rt.fake_elapsed(1.0)
        self.rt.fake_pause(0)
        self.rt.fake_hold(0)
        self.rt.fake_clear()
        self.rt.fake_call(0)

    def stream(self) -> int:
        s = ctypes.c_void_p()
        self.rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1)
        return s.value

    def malloc(self, nbytes: int) -> int:
        p = ctypes.c_void_p()
        assert self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(nbytes)) == 0
        return p.value

    def blocks(self) -> set[int]:
        a = (ctypes.c_uint64 * 4096)()
        return set(a[:self.rt.fake_blocks(a, 4096)])

    def call(self, i: int):
        self.rt.fake_call(i)

    def ops(self) -> list[Op]:
        return [Op(o["call"], o["stream"], o["index"], o["name"], o["dst"], o["bytes"], tuple(o["arg"]),
                   {int(k): v for k, v in o["seen"].items()}) for o in json.loads(self.rt.fake_ops())]

    def begin_capture(self, stream: int, mode: int):
        assert self.rt.cudaStreamBeginCapture(ctypes.c_void_p(stream), mode) == 0

    def end_capture(self, stream: int) -> int:
        g = ctypes.c_void_p()
        return self.rt.cudaStreamEndCapture(ctypes.c_void_p(stream), ctypes.byref(g))
