"""The library's host side on a stand-in for the CUDA runtime (tests/cpp/fake_cudart.cpp): no GPU, kernels do
nothing, and any runtime call can be made to fail."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np

from conftest import ROOT


def build(out_dir, sources=("ta3s_surrogate.cu", "ta3s_wide.cu")) -> C.CDLL:
    from tetris_ai3_b200 import build as b
    from tetris_ai3_b200 import evaluator, surrogate
    so = os.path.join(str(out_dir), "libfake_%s.so" % sources[0].split(".")[0])
    # the kernels never run: PTX alone, without the assembler's minute
    subprocess.run([b.nvcc(), "-gencode", "arch=compute_100a,code=compute_100a", "-O1", "-std=c++20", "-fmad=false",
                    "-Xcompiler", "-fPIC", "-shared", "-Xlinker", "-Bsymbolic",     # (torch's runtime may be loaded too)
                    "--expt-relaxed-constexpr", "-cudart", "none",
                    "-I", os.path.join(ROOT, "include"), "-I", b.CSRC, "-o", so,
                    *(os.path.join(b.CSRC, s) for s in sources),
                    os.path.join(ROOT, "tests", "cpp", "fake_cudart.cpp")], check=True)
    if "ta3b_eval.cu" in sources:
        lib = evaluator.library(so)
    else:
        lib = C.CDLL(so)
        for name, (res, args) in surrogate._SIG.items():
            f = getattr(lib, name)
            f.restype, f.argtypes = res, args
    lib.fake_block.restype = C.c_void_p
    lib.fake_block.argtypes = [C.c_size_t]
    lib.fake_capture.argtypes = [C.c_char_p, C.c_int, C.c_size_t]
    lib.fake_log.restype, lib.fake_log.argtypes = C.c_size_t, [C.c_char_p, C.c_size_t]
    lib.fake_arg.restype = C.c_size_t
    return lib


def _p(a):
    return None if a is None else C.c_void_p(a.ctypes.data)


class Model:
    """One surrogate (kind "ta3s", 97 inputs, or "ta3w") through its C interface; calls return their status."""

    def __init__(self, lib, kind: str, in_dim: int = 97, hidden: int = 128):
        self.lib, self.kind, self.in_dim = lib, kind, in_dim
        self.h = lib.ta3s_create(0, 1) if kind == "ta3s" else lib.ta3w_create(0, in_dim, hidden, 1)
        assert self.h
        self.nparam = lib.ta3s_num_params() if kind == "ta3s" else lib.ta3w_model_params(self.h)

    def f(self, name):
        return getattr(self.lib, f"{self.kind}_{name}")

    def close(self):
        self.f("destroy")(self.h)

    def error(self) -> str:
        return self.f("last_error")(self.h).decode()

    def set_data(self, rows: int, name="set_data"):
        x = np.random.default_rng(rows).standard_normal((rows, self.in_dim), dtype=np.float32)
        y = x[:, 0].copy()
        return self.f(name)(self.h, _p(x), _p(y), rows)

    def gradients(self):
        g = np.zeros(self.nparam, np.float32)
        return self.f("gradients")(self.h, _p(g), None)

    def train(self, epochs: int, batch: int):
        return self.f("train")(self.h, epochs, batch, 1e-3, 0.0, 0, None)

    def predict(self, rows: int):
        x, mean = np.zeros((rows, self.in_dim), np.float32), np.zeros(rows, np.float32)
        return self.f("predict")(self.h, _p(x), rows, _p(mean), None)

    # the stand-in
    def log(self) -> list[str]:
        buf = C.create_string_buffer(1 << 20)
        self.lib.fake_log(buf, len(buf))
        return buf.value.decode().split()

    def launches(self, kernel: str) -> int:
        return self.lib.fake_count(kernel.encode())

    def captured(self, dtype, nth: int = 0):
        """The captured argument's bytes in the nth launch (fake_capture)."""
        buf = np.zeros(4096, np.uint8)
        return buf[:self.lib.fake_arg(nth, _p(buf))].view(dtype)
