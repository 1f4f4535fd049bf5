"""The Python methods and the extension module in front of the C ABI, run without a GPU: a library of the same name whose
entry points only write their arguments down, and tensors that say they are on cuda:0 but have no memory behind them (nothing
reads it).  A call that reaches an entry point here is a launch there.

Runs in a process of its own: the extension resolves libsiglip_fp8.so by name, and must not meet the real one.
    python -m tests.fake_abi <folder> <module> <table>      prints {case: {route: [error, message, calls]}} as JSON
"""
from __future__ import annotations

import ctypes as C
import importlib
import itertools
import json
import os
import shutil
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
STREAM = 77       # the stream every case names: torch's current one needs a driver

_CTYPE = {C.c_void_p: "void*", C.c_int: "int", C.c_int64: "long long", C.c_uint: "unsigned", C.c_float: "float", C.c_char_p: "const char*"}
_SPECIAL = {"sl8_create": "*(void**)a0 = (void*)0x1000; return 0;", "sl8_destroy": "return 0;", "sl8_last_error_string": 'return "";',
            "sl8_version": 'return "";', "sl8_padded_table_rows": "return a0 + 127;",
            "sl8_linear_bias_fp8": f"return sl8_fc1_gelu_fp8({', '.join(f'a{i}' for i in range(15))}, a15 | 4, a16);"}


def source(signatures: dict) -> str:
    out = ["#include <stdio.h>", "#include <string.h>", "static char text[1 << 16];", "static int used;",
           "const char* fake_calls(void) { text[used] = 0; used = 0; return text; }"]
    for name, (res, args) in signatures.items():
        types = [_CTYPE.get(a, "void*") for a in args]
        head = f"{_CTYPE[res]} {name}({', '.join(f'{t} a{i}' for i, t in enumerate(types)) or 'void'})"
        if name in _SPECIAL:
            out.append(f"{head} {{ {_SPECIAL[name]} }}")
            continue
        show = [("%.9g", f"(double)a{i}") if t == "float" else ("%lld", f"(long long)a{i}") for i, t in enumerate(types)]
        fmt = " ".join([name] + [f for f, _ in show])
        out.append(f'{head} {{ used += snprintf(text + used, sizeof text - used, "{fmt}\\n"{"".join(", " + a for _, a in show)}); return 0; }}')
    return "\n".join(out)


def install(folder: Path) -> None:
    """The recording library and a copy of the extension module, side by side in `folder`."""
    from siglip_b200 import build, lib
    build.build()
    src = folder / "fake.c"
    src.write_text(source(lib.SIGNATURES))
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", str(folder / "libsiglip_fp8.so"), str(src)], check=True)
    shutil.copy(build.BINDING, folder / build.BINDING.name)


def run_child(folder: Path, module: str, table: str, **env) -> subprocess.CompletedProcess:
    return subprocess.run([sys.executable, "-m", "tests.fake_abi", str(folder), module, table], cwd=ROOT, capture_output=True, text=True,
                          timeout=600, env={**os.environ, **env})


_next = itertools.count(1)


def cuda(*shape, dtype=None, stride=None, elements=None, offset=0, device=0):
    """A tensor on cuda:`device` of that shape (contiguous unless `stride` is given) at an address of its own; its storage holds
    `elements` elements (what the shape spans unless given)."""
    import torch
    dtype = torch.uint8 if dtype is None else dtype
    if stride is None:
        stride = [1]
        for n in reversed(shape[1:]):
            stride.insert(0, stride[0] * max(n, 1))
    span = offset + (0 if 0 in shape else 1 + sum((n - 1) * s for n, s in zip(shape, stride)))
    at = torch.device("cuda", device)
    storage = torch._C._construct_storage_from_data_pointer(next(_next) << 32, at, (span if elements is None else elements) * dtype.itemsize)
    return torch._C._construct_CUDA_Tensor_From_Storage_And_Metadata(
        {"size": shape, "stride": tuple(stride), "dtype": dtype, "device": at, "storage_offset": offset}, storage)


def engines(folder: Path):
    """(an engine whose calls go through the extension, one whose calls stay in Python, what takes the calls written down)."""
    import siglip_b200
    from siglip_b200 import lib
    lib._LIB_PATH, lib._BINDING_PATH = folder / "libsiglip_fp8.so", folder / "sl8_torch.so"
    library = C.CDLL(str(lib._LIB_PATH))
    library.fake_calls.restype = C.c_char_p
    fast, slow = siglip_b200.Engine(0), siglip_b200.Engine(0)
    slow._native = lib.NoBinding()
    return fast, slow, lambda: library.fake_calls().decode().splitlines()


def main(folder: str, module: str, table: str) -> None:
    from tests import fake_abi
    cases = getattr(importlib.import_module(module), table)
    fast, slow, taken = engines(Path(folder))
    out = {}
    for name, case in cases.items():
        out[name] = {}
        for route, engine in (("extension", fast), ("python", slow)):
            fake_abi._next = itertools.count(1)        # the same addresses on both routes
            error = message = None
            try:
                case(engine)
            except Exception as e:
                error, message = type(e).__name__, str(e)
            out[name][route] = [error, message, taken()]
    print(json.dumps(out))


if __name__ == "__main__":
    main(*sys.argv[1:])
