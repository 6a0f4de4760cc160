"""ctypes binding of ``libclt_b200.so``.

The argument types of every entry point are read from ``include/clt_b200.h`` so the
binding cannot drift from the declared C ABI.  There is no fallback: when the
library is missing, cannot be loaded, or the current device is not sm_100, the
first use raises.
"""
from __future__ import annotations

import ctypes
import importlib.machinery
import importlib.util
import re
import sysconfig
from pathlib import Path
from typing import Dict, List, Tuple

import torch

PKG = Path(__file__).resolve().parent
HEADER = PKG.parent / "include" / "clt_b200.h"
LIB_PATH = PKG / "libclt_b200.so"
#: The name carries the interpreter's ABI tag: a tree built under one Python and imported under another has none.
BINDING_PATH = PKG / ("_clt_call" + (sysconfig.get_config_var("EXT_SUFFIX") or ".so"))

_CTYPES = {
    "int": ctypes.c_int,
    "float": ctypes.c_float,
    "int64_t": ctypes.c_int64,
    "clt_stream_t": ctypes.c_void_p,
}


def parse_header(path: Path = HEADER) -> Dict[str, Tuple[object, List[Tuple[str, object]]]]:
    """{name: (restype, [(argname, ctype), ...])} for every ``clt_*`` prototype."""
    text = re.sub(r"/\*.*?\*/", "", path.read_text(), flags=re.S)
    protos = {}
    for m in re.finditer(r"(const\s+char\s*\*|int)\s+(clt_\w+)\s*\(([^)]*)\)\s*;", text):
        ret, name, args = m.group(1), m.group(2), m.group(3).strip()
        restype = ctypes.c_char_p if "char" in ret else ctypes.c_int
        arglist = []
        if args and args != "void":
            for a in args.split(","):
                a = " ".join(a.split())
                if "*" in a:
                    arglist.append((a.split("*")[-1].strip(), ctypes.c_void_p))
                else:
                    typ, an = a.rsplit(" ", 1)
                    arglist.append((an, _CTYPES[typ.replace("const ", "").strip()]))
        protos[name] = (restype, arglist)
    return protos


class CltError(RuntimeError):
    pass


class _Lib:
    def __init__(self):
        if not LIB_PATH.exists():
            raise CltError(
                f"{LIB_PATH} is missing: build it with `python -m crosslayer_transcoder_b200.build` "
                "(there is no CPU or PyTorch fallback)")
        self.cdll = ctypes.CDLL(str(LIB_PATH))
        self.protos = parse_header()
        self._fn = {}
        for name, (restype, args) in self.protos.items():
            fn = getattr(self.cdll, name)          # AttributeError if a declared symbol is not exported
            fn.restype = restype
            fn.argtypes = [t for _, t in args]
            self._fn[name] = fn
        self._native = self._bind_native()
        self._device_ok = set()

    def _bind_native(self):
        """{name: wrapper} of the compiled call path (``build.binding_source``), empty where it was not built, does not
        load, or was built from other prototypes or conversions: calls then go through ctypes."""
        from .build import binding_source

        if not BINDING_PATH.exists():
            return {}
        loader = importlib.machinery.ExtensionFileLoader("_clt_call", str(BINDING_PATH))
        try:
            mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("_clt_call", loader))
            loader.exec_module(mod)
        except ImportError:
            return {}
        if getattr(mod, "source", None) != binding_source(self.protos)[0]:
            return {}
        return {n: getattr(mod, n) for n, fn in self._fn.items()
                if hasattr(mod, n) and mod.bind(n, ctypes.cast(fn, ctypes.c_void_p).value)}

    def last_error(self) -> str:
        s = self.cdll.clt_last_error()
        return s.decode() if s else ""

    def check_device(self):
        # (a device that has been checked is there: asking the driver again cost as much as a launch)
        if not self._device_ok and not torch.cuda.is_available():
            raise CltError("no CUDA device: this package runs on B200 (sm_100a) only and has no CPU fallback")
        dev = torch.cuda.current_device()
        if dev not in self._device_ok:
            if self.cdll.clt_device_check() != 0:
                raise CltError(self.last_error())
            self._device_ok.add(dev)

    def query(self, name: str, *args) -> int:
        """The value of an entry point that launches nothing and cannot fail."""
        return (self._native.get(name) or self._fn[name])(*args)

    def call(self, name: str, *args):
        """Call an ``int``-returning entry point; tensors are passed as their data pointers."""
        native = self._native.get(name)
        rc = None
        if native is not None:
            try:
                rc = native(*args)
            except TypeError:
                pass            # nothing was called: ctypes takes its own pointer objects, or says what is wrong
        if rc is None:
            rc = self._fn[name](*[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args])
        if rc != 0:
            raise CltError(f"{name} failed ({rc}): {self.last_error()}")


_lib = None


def lib() -> _Lib:
    global _lib
    if _lib is None:
        _lib = _Lib()
    return _lib


def stream_ptr() -> int:
    """The current stream's handle, without the Stream object (5 us a call, five calls a step)."""
    if not torch.cuda.is_initialized():
        torch.cuda.init()
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


DTYPE_CODE = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}

STATUS_NAMES = {
    0x10: "the MMA warp gave up waiting for a TMA stage",
    0x11: "the TMA warp gave up waiting for a free stage",
    0x12: "the epilogue gave up waiting for an accumulator",
    0x13: "the MMA warp gave up waiting for the epilogue",
    0x20: "an index read from memory was out of range",
    0x21: "a fixed-capacity list overflowed",
}


def check_status(status: torch.Tensor, where: str = ""):
    """Read the device status word (synchronises) and raise if a kernel reported a failure."""
    code = int(status.item())
    if code != 0:
        status.zero_()
        raise CltError(f"device status {code:#x} {where}: {STATUS_NAMES.get(code, 'unknown code')}")
