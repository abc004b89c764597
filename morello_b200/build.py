"""Builds the CUDA extension (the C-ABI shared library) in-tree for sm_100a."""
import os
import shutil
import subprocess
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB_DIR = os.path.join(HERE, "_lib")
LIB_PATH = os.path.join(LIB_DIR, "libmorello_b200.so")
SOURCES = ["combine.cu", "devplan.cu", "plan.cpp", "optable.cpp", "capi.cpp"]
# The Python mirror's query calls (CPython C API); loaded as morello_b200._lib's helper, not as a package. The
# name carries the interpreter's ABI, so that one built for another interpreter is not taken.
PYHOST_PATH = os.path.join(LIB_DIR, "_pyhost" + sysconfig.get_config_var("EXT_SUFFIX"))


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found; the CUDA extension cannot be built")
    return nvcc


def _has_python_headers():
    return os.path.exists(os.path.join(sysconfig.get_paths()["include"], "Python.h"))


def needs_build():
    targets = [LIB_PATH] + ([PYHOST_PATH] if _has_python_headers() else [])
    if not all(os.path.exists(t) for t in targets):
        return True
    built = min(os.path.getmtime(t) for t in targets)
    deps = []
    for root, _dirs, files in os.walk(CSRC):
        deps += [os.path.join(root, f) for f in files]
    deps.append(os.path.join(HERE, "..", "include", "morello_b200.h"))
    return any(os.path.getmtime(d) > built for d in deps if os.path.exists(d))


def build(force=False, verbose=False):
    """nvcc -gencode arch=compute_100a,code=sm_100a ... -shared -> morello_b200/_lib/. The helper of the
    Python mirror's query calls needs the interpreter's headers; without them it is left out, and the mirror
    packs its queries in Python."""
    if not force and not needs_build():
        return LIB_PATH
    os.makedirs(LIB_DIR, exist_ok=True)
    cmd = [
        _nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
        "-Xcompiler", "-fPIC,-pthread,-Wno-stringop-overflow", "-shared", "-o", LIB_PATH,
    ] + [os.path.join(CSRC, s) for s in SOURCES]
    if verbose:
        cmd.insert(1, "-Xptxas")
        cmd.insert(2, "-v")
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
        raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    if _has_python_headers():
        res = subprocess.run([_nvcc(), "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I" + sysconfig.get_paths()["include"],
                              os.path.join(CSRC, "pyhost.cpp"), "-o", PYHOST_PATH], capture_output=True, text=True)
        if res.returncode != 0:
            raise RuntimeError("nvcc failed:\n" + res.stdout + res.stderr)
    return LIB_PATH
