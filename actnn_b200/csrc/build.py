"""Build ``libactnn_b200.so`` in-tree with nvcc for sm_100a.

    python -m actnn_b200.csrc.build          (or: python actnn_b200/csrc/build.py)

The library is plain CUDA behind a C ABI (``include/actnn_b200.h``), no torch headers involved; the
binding's C++ half (``native.cpp``) is built beside it.  Objects are compiled in parallel and cached by mtime.
"""
from __future__ import annotations

import os
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCES = ["api.cu", "codec_mixed.cu", "codec_single.cu", "codec_generic.cu", "codec_column.cu", "codec_ragged.cu",
           "compress_mixed.cu", "stats.cu", "mask_ops.cu",
           "maxpool.cu", "batch_norm.cu", "bn_column.cu", "layout.cu"]
HEADERS = ["common.cuh", "quant_math.cuh", "mixed_bundle.cuh", "column.cuh", "flat_runs.cuh", os.path.join("..", "..", "include", "actnn_b200.h")]
LIB = os.path.join(HERE, "libactnn_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
         "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _stale(target: str, deps) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(verbose: bool = False, force: bool = False) -> str:
    headers = [os.path.join(HERE, h) for h in HEADERS] + [os.path.abspath(__file__)]
    jobs = []
    objs = []
    for src in SOURCES:
        s = os.path.join(HERE, src)
        o = os.path.join(HERE, src.replace(".cu", ".o"))
        objs.append(o)
        if force or _stale(o, [s] + headers):
            cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", s, "-o", o]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("nvcc failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
        return r.stderr

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for out in ex.map(run, jobs):
            if verbose and out:
                print(out)
    if jobs or force or _stale(LIB, objs):
        run([NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a",
                                                   "-cudart", "shared"])
    build_fastcall(force)
    build_native(force)
    return LIB


# ---------------------------------------------------------------------------------------
# Fast call path for the Python binding: a small CPython module with one METH_FASTCALL wrapper
# per entry point, generated from the signature table (actnn_b200/_signatures.py).  ctypes
# spends ~10 microseconds marshalling the 12-25 arguments of a call; at ~500 calls per training
# step of a ResNet-50 that is a tenth of the step.  The wrappers take the same arguments
# (ints, floats, None for a null pointer) and return the status.
# ---------------------------------------------------------------------------------------
FAST_SRC = os.path.join(HERE, "_actnn_fastcall.c")
FAST_LIB = os.path.join(HERE, "_actnn_fastcall.so")
_C_TYPE = {"P": "void*", "I": "int", "L": "long long", "U": "unsigned long long", "F": "float", "D": "double"}
_C_CONV = {"P": "as_ptr(a[%d])", "I": "(int)PyLong_AsLong(a[%d])", "L": "PyLong_AsLongLong(a[%d])",
           "U": "PyLong_AsUnsignedLongLongMask(a[%d])", "F": "(float)PyFloat_AsDouble(a[%d])",
           "D": "PyFloat_AsDouble(a[%d])"}


def _signatures():
    import importlib.util
    spec = importlib.util.spec_from_file_location("_actnn_signatures", os.path.join(HERE, "..", "_signatures.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod.SIGNATURES


def generate_fastcall_source() -> str:
    out = ["/* Generated by actnn_b200/csrc/build.py from actnn_b200/_signatures.py: do not edit. */",
           "#define PY_SSIZE_T_CLEAN", "#include <Python.h>", "",
           "static void* as_ptr(PyObject* o) {",
           "  if (o == Py_None) return NULL;",
           "  return (void*)PyLong_AsUnsignedLongLongMask(o);", "}", ""]
    table = []
    for name, letters in _signatures().items():
        out.append("extern int %s(%s);" % (name, ", ".join(_C_TYPE[c] for c in letters)))
        out.append("static PyObject* f_%s(PyObject* self, PyObject* const* a, Py_ssize_t n) {" % name)
        out.append("  if (n != %d) { PyErr_SetString(PyExc_TypeError, \"%s expects %d arguments\"); return NULL; }"
                   % (len(letters), name, len(letters)))
        for i, c in enumerate(letters):
            out.append("  %s v%d = %s;" % (_C_TYPE[c], i, _C_CONV[c] % i))
        out.append("  if (PyErr_Occurred()) return NULL;")
        out.append("  return PyLong_FromLong(%s(%s));" % (name, ", ".join("v%d" % i for i in range(len(letters)))))
        out.append("}")
        table.append('  {"%s", (PyCFunction)(void (*)(void))f_%s, METH_FASTCALL, NULL},' % (name, name))
    out += ["", "static PyMethodDef methods[] = {"] + table + ["  {NULL, NULL, 0, NULL}", "};",
            'static struct PyModuleDef module = {PyModuleDef_HEAD_INIT, "_actnn_fastcall", NULL, -1, methods};',
            "PyMODINIT_FUNC PyInit__actnn_fastcall(void) { return PyModule_Create(&module); }", ""]
    return "\n".join(out)


def build_fastcall(force: bool = False) -> str:
    import sysconfig
    src = generate_fastcall_source()
    if not os.path.exists(FAST_SRC) or open(FAST_SRC).read() != src:
        with open(FAST_SRC, "w") as f:
            f.write(src)
    if force or _stale(FAST_LIB, [FAST_SRC, LIB]):
        cmd = [os.environ.get("CC", "gcc"), "-O2", "-shared", "-fPIC", "-I" + sysconfig.get_paths()["include"],
               FAST_SRC, "-o", FAST_LIB, "-L" + HERE, "-lactnn_b200", "-Wl,-rpath,$ORIGIN"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("gcc failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
    return FAST_LIB


# ---------------------------------------------------------------------------------------
# The host side of the hot entry points (native.cpp): the only source that needs torch's headers.
# ---------------------------------------------------------------------------------------
NATIVE_SRC = os.path.join(HERE, "native.cpp")
NATIVE_LIB = os.path.join(HERE, "_actnn_native.so")


def build_native(force: bool = False) -> str:
    if not force and not _stale(NATIVE_LIB, [NATIVE_SRC, os.path.join(HERE, HEADERS[-1]), os.path.abspath(__file__)]):
        return NATIVE_LIB
    import sysconfig

    import torch
    from torch.utils import cpp_extension as ext
    # the system compiler, whatever CXX says: the module must share libstdc++.so.6 with torch, and a compiler that
    # links its own copy statically makes a module that crashes when a number is formatted
    cmd = ["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-O2", "-std=c++17", "-shared", "-fPIC", NATIVE_SRC, "-o", NATIVE_LIB,
           "-DTORCH_EXTENSION_NAME=_actnn_native", "-DTORCH_API_INCLUDE_EXTENSION_H",
           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
           "-I" + sysconfig.get_paths()["include"], "-I/usr/local/cuda/include"]
    cmd += ["-isystem" + d for d in ext.include_paths()]
    libdir = os.path.join(os.path.dirname(torch.__file__), "lib")
    cmd += ["-L" + libdir, "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda", "-ltorch", "-ltorch_python",
            "-L" + HERE, "-lactnn_b200", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("g++ failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
    return NATIVE_LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv, force="-f" in sys.argv))
