"""Build ``libclt_b200.so`` (the CUDA kernels behind the C ABI of ``include/clt_b200.h``)
in-tree with nvcc for sm_100a.  ``python -m crosslayer_transcoder_b200.build`` rebuilds it."""
from __future__ import annotations

import ctypes
import hashlib
import os
import shutil
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
LIB = PKG / "libclt_b200.so"
OBJ = PKG / "build"

NVCC_FLAGS = ["-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC", "--use_fast_math=false"]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and Path(cand).exists():
            return cand
    raise RuntimeError("nvcc not found; set NVCC or add it to PATH")


def _stale(target: Path, deps) -> bool:
    if not target.exists():
        return True
    t = target.stat().st_mtime
    return any(Path(d).stat().st_mtime > t for d in deps)


# ---- native call path -------------------------------------------------------------------------------------------
# One wrapper per int-returning prototype of the header, so that a call from Python converts its arguments in C
# (about 1 us instead of the 9 us of a 17-argument call through ctypes).
_C_PRELUDE = r"""
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <stdint.h>

static PyObject* s_data_ptr;

static int as_ptr(PyObject* a, void** out) {
  if (a == Py_None) { *out = 0; return 1; }
  if (!PyLong_Check(a)) {
    PyObject* p = PyObject_CallMethodNoArgs(a, s_data_ptr);
    if (!p) {
      if (PyErr_ExceptionMatches(PyExc_AttributeError)) {
        PyErr_Clear();
        PyErr_SetString(PyExc_TypeError, "expected None, an address or a tensor");
      }
      return 0;
    }
    *out = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(p);
    Py_DECREF(p);
    return !PyErr_Occurred();
  }
  *out = (void*)(uintptr_t)PyLong_AsUnsignedLongLongMask(a);
  return !PyErr_Occurred();
}
static int as_i64(PyObject* a, int64_t* out) {
  if (!PyLong_Check(a)) { PyErr_SetString(PyExc_TypeError, "expected an integer"); return 0; }
  *out = (int64_t)PyLong_AsUnsignedLongLongMask(a);
  return !PyErr_Occurred();
}
static int as_f32(PyObject* a, float* out) {
  if (!PyFloat_Check(a) && !PyLong_Check(a)) { PyErr_SetString(PyExc_TypeError, "expected a number"); return 0; }
  *out = (float)PyFloat_AsDouble(a);
  return !PyErr_Occurred();
}
"""


def binding_source(protos):
    """(digest, text): C source of the ``_clt_call`` extension module for ``_lib.parse_header``'s prototypes.
    ``bind(name, address)`` gives a wrapper its entry point; a wrapper raises TypeError before it calls anything.  The
    module's ``source`` is the digest, so that one which was made from another text is recognised."""
    kinds = {ctypes.c_void_p: ("void*", "void*", "as_ptr"), ctypes.c_int: ("int", "int64_t", "as_i64"),
             ctypes.c_int64: ("int64_t", "int64_t", "as_i64"), ctypes.c_float: ("float", "float", "as_f32")}
    names = [n for n, (ret, args) in protos.items() if ret is ctypes.c_int and args]
    out = [_C_PRELUDE]
    for i, name in enumerate(names):
        types = [kinds[t] for _, t in protos[name][1]]
        out.append(f"static int (*f{i})({', '.join(t[0] for t in types)});")
        out.append(f"static PyObject* w{i}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{")
        out.append(f'  if (!f{i}) {{ PyErr_SetString(PyExc_RuntimeError, "{name} is not bound"); return 0; }}')
        out.append(f'  if (n != {len(types)}) return PyErr_Format(PyExc_TypeError, "{name}: %zd arguments, expected '
                   f'{len(types)}", n);')
        for j, t in enumerate(types):
            out.append(f"  {t[1]} v{j}; if (!{t[2]}(a[{j}], &v{j})) return 0;")
        call = ", ".join(f"({t[0]})v{j}" for j, t in enumerate(types))
        out.append(f"  int rc; Py_BEGIN_ALLOW_THREADS rc = f{i}({call}); Py_END_ALLOW_THREADS")
        out.append("  return PyLong_FromLong(rc);\n}")
    out.append("static void** const slots[] = {" + ", ".join(f"(void**)&f{i}" for i in range(len(names))) + "};")
    out.append("static const char* const slot_names[] = {" + ", ".join(f'"{n}"' for n in names) + "};")
    out.append("""static PyObject* bind(PyObject* self, PyObject* args) {
  const char* name; unsigned long long addr;
  if (!PyArg_ParseTuple(args, "sK", &name, &addr)) return 0;
  for (size_t i = 0; i < sizeof(slots) / sizeof(slots[0]); ++i)
    if (strcmp(slot_names[i], name) == 0) { *slots[i] = (void*)(uintptr_t)addr; Py_RETURN_TRUE; }
  Py_RETURN_FALSE;
}""")
    out.append('static PyMethodDef methods[] = {{"bind", bind, METH_VARARGS, 0},')
    out += [f'  {{"{n}", (PyCFunction)(void*)w{i}, METH_FASTCALL, 0}},' for i, n in enumerate(names)]
    out.append("  {0}};\nstatic struct PyModuleDef def = {PyModuleDef_HEAD_INIT, \"_clt_call\", 0, -1, methods};")
    out.append('PyMODINIT_FUNC PyInit__clt_call(void) {\n  s_data_ptr = PyUnicode_InternFromString("data_ptr");\n'
               '  PyObject* m = s_data_ptr ? PyModule_Create(&def) : 0;\n'
               '  if (m) PyModule_AddStringConstant(m, "source", SOURCE);\n'
               '  return m;\n}\n')
    text = "\n".join(out)
    digest = hashlib.sha256(text.encode()).hexdigest()
    return digest, f'#define SOURCE "{digest}"\n{text}'


def _binding_tools():
    """(folder of Python's headers, C compiler), None for what this host does not have."""
    include = sysconfig.get_paths()["include"]
    return include if (Path(include) / "Python.h").exists() else None, shutil.which("gcc") or shutil.which("cc")


def build_binding(force: bool = False):
    """Compile the native call path.  Without Python's headers there is none, and calls go through ctypes."""
    from ._lib import BINDING_PATH, parse_header

    include, cc = _binding_tools()
    if include is None or cc is None:
        BINDING_PATH.unlink(missing_ok=True)
        return None
    src, (_, text) = OBJ / "clt_call.c", binding_source(parse_header())
    if force or not src.exists() or src.read_text() != text or _stale(BINDING_PATH, [src]):
        OBJ.mkdir(exist_ok=True)
        src.write_text(text)
        cmd = [cc, "-O2", "-shared", "-fPIC", f"-I{include}", str(src), "-o", str(BINDING_PATH)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"{cc} failed on {src.name}:\n{r.stderr}")
    return BINDING_PATH


def build(force: bool = False, verbose: bool = False) -> Path:
    nvcc = _nvcc()
    flags = [f for f in NVCC_FLAGS if not f.startswith("--use_fast_math")]
    headers = sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.h")) + sorted((PKG.parent / "include").glob("*.h"))
    sources = sorted(CSRC.glob("*.cu"))
    OBJ.mkdir(exist_ok=True)
    jobs = []
    for src in sources:
        obj = OBJ / (src.stem + ".o")
        if force or _stale(obj, [src, *headers]):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc, *flags, "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src.name}:\n{r.stdout}\n{r.stderr}")
        return r.stderr

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for out in ex.map(compile_one, jobs):
            if verbose and out:
                print(out)
    objs = [OBJ / (s.stem + ".o") for s in sources]
    if force or jobs or _stale(LIB, objs):
        cmd = [nvcc, "-shared", "-o", str(LIB), *map(str, objs), "-gencode", "arch=compute_100a,code=sm_100a",
               "-cudart", "static"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    build_binding(force)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
