"""The C ABI's host code (csrc/api.cu) on a stand-in CUDA runtime (fake_cuda.cpp)."""
import ctypes
import os
import re
import subprocess
from pathlib import Path

import numpy as np

from phonomena_gb300 import _lib, build

HERE = Path(__file__).resolve().parent


def compile_host_abi():
    """api.cu with its two counter launches replaced, and fake_cuda.cpp, by the host compiler."""
    out = HERE / "_build"
    out.mkdir(exist_ok=True)
    text, n = re.subn(r"\w+<<<1, 1, 0, (.+?)>>>\(.*?\);", r"fake_launch(\1);", (build.CSRC / "api.cu").read_text())
    assert n > 0 and "<<<" not in text
    src = out / "host_abi.cpp"
    src.write_text('#include "fake_prelude.h"\n' + text.replace("../../include/", ""))
    lib = out / f"libhost_abi.{os.getpid()}.so"
    cuda = Path(build.nvcc()).resolve().parents[1] / "include"
    # (-Bsymbolic: a CUDA runtime that the process has loaded, as torch does, must not take the calls)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic",
                    "-I", str(cuda), "-I", str(HERE), "-I", str(build.CSRC), "-I", str(build.ROOT / "include"), str(src),
                    str(HERE / "fake_cuda.cpp"), "-o", str(lib)], check=True)
    L = ctypes.CDLL(str(lib))
    lib.unlink()
    vp, ci, sz = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
    for name, res, args in (("phono_create", ci, [vp, vp]), ("phono_destroy", None, [vp]), ("phono_stream", vp, [vp]),
                            ("phono_set_source", ci, [vp, vp, ci]), ("phono_step", ci, [vp, ci]),
                            ("phono_set_materials", ci, [vp, vp, vp, ci]), ("phono_download_materials", ci, [vp, vp, sz]),
                            ("phono_download", ci, [vp, ci, vp, sz]), ("phono_upload", ci, [vp, ci, vp, sz]),
                            ("phono_set_tiling", ci, [vp, ci, ci]), ("phono_last_error", ctypes.c_char_p, []),
                            ("phono_footprint", ci, [ci] * 6 + [vp]), ("phono_footprint_shaped", ci, [ci] * 8 + [vp]),
                            ("phono_batch_create", ci, [ci, ci, ci, vp]), ("phono_batch_add", ci, [vp, vp, ci]),
                            ("phono_batch_remove", ci, [vp, ci]), ("phono_batch_step", ci, [vp, ci]),
                            ("phono_batch_sync", ci, [vp]), ("phono_batch_destroy", None, [vp]),
                            ("fake_reset", None, []), ("fake_limit", None, [sz]), ("fake_hold", None, [vp, ci]), ("fake_fail", None, [ctypes.c_char_p, ci]),
                            ("fake_device", None, [ci]), ("fake_current", ci, []), ("fake_broken", ci, []),
                            ("fake_count", ci, [ctypes.c_char_p]), ("fake_bytes", sz, [ci]), ("fake_pin", None, [vp, sz])):
        f = getattr(L, name)
        f.restype, f.argtypes = res, args
    return L


TABLE = np.array([[224e9, 64e9, 64e9, 64e9, 224e9, 64e9, 64e9, 64e9, 224e9, 80e9, 80e9, 80e9, 2330.0]] * 4)


class Handle:
    """A handle of uniform spacing; calls return the C ABI's codes."""

    def __init__(self, L, shape, precision="f32k", max_steps=100, tile_j=0, x_segment=0, seed=0, record_every=0):
        self.L, self.shape = L, shape
        self.ids = np.random.default_rng(seed).integers(0, len(TABLE), shape, dtype=np.uint8)
        arrs = [np.full(n - d, 1e-5) for d in (1, 2) for n in shape]
        d = _lib.PhonoDesc(*shape, *(a.ctypes.data for a in arrs), self.ids.ctypes.data, TABLE.ctypes.data, len(TABLE), 1e-10,
                           _lib.PRECISIONS[precision], 1, 0, 0, max_steps, record_every, tile_j, x_segment)
        h = ctypes.c_void_p()
        self.rc = L.phono_create(ctypes.byref(d), ctypes.byref(h))
        self.h = h
        if self.rc == 0:
            src = np.zeros(max_steps)
            assert L.phono_set_source(h, src.ctypes.data, max_steps) == 0

    def set_ids(self, seed):
        self.ids = np.random.default_rng(seed).integers(0, len(TABLE), self.shape, dtype=np.uint8)
        return self.L.phono_set_materials(self.h, self.ids.ctypes.data, TABLE.ctypes.data, len(TABLE))

    def ids_arrived(self):
        got = np.empty(self.shape, np.uint8)
        assert self.L.phono_download_materials(self.h, got.ctypes.data, got.nbytes) == 0
        return np.array_equal(got, self.ids)

    def stream(self):
        return self.L.phono_stream(self.h)

    def close(self):
        self.L.phono_destroy(self.h)
