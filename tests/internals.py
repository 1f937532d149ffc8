"""Addresses of device words that the C ABI does not hand out, for tests that
set them or look at them: a small library compiled against csrc/hg_internal.h."""
import ctypes as C
import os
import subprocess
import tempfile
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]

SOURCE = """
#include "hg_internal.h"
extern "C" {
void* error_word(hg_ctx* ctx) { return ctx->err; }
void* moments(hg_mlp* mlp, int which) { return which ? mlp->adam_v : mlp->adam_m; }
}
"""


def load() -> C.CDLL:
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    with tempfile.TemporaryDirectory() as d:
        src, lib = Path(d) / "internals.cpp", Path(d) / "internals.so"
        src.write_text(SOURCE)
        subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{ROOT / 'bevy_hair_gb300' / 'csrc'}",
                        f"-I{cuda}/include", "-o", str(lib), str(src)], check=True)
        out = C.CDLL(str(lib))
    out.error_word.restype = out.moments.restype = C.c_void_p
    out.error_word.argtypes = [C.c_void_p]
    out.moments.argtypes = [C.c_void_p, C.c_int]
    return out


def device_words(address: int, count: int):
    """`count` 32-bit words at a device address, as a torch tensor."""
    import torch

    class Words:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "version": 2, "data": (address, False)}

    return torch.as_tensor(Words(), device="cuda")
