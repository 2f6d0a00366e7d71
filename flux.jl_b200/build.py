"""Builds libfluxb200.so (hand-written CUDA for sm_100a + the C ABI) in-tree with nvcc.

    python flux.jl_b200/build.py [--force] [--verbose]

Each csrc/*.cu is compiled to an object file (in parallel) and linked into
fluxb200/libfluxb200.so; native Python wrappers of its entry points are generated from the header
(fluxb200/_fastcall*.so).  The CUDA runtime is linked statically and the driver API is reached
through cudaGetDriverEntryPoint, so the library also loads on a machine without a GPU driver
(where every compute entry point reports FB_ERR_CUDA).
"""
from __future__ import annotations

import concurrent.futures
import os
import re
import shutil
import subprocess
import sys
import sysconfig

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
OUT = os.path.join(HERE, "fluxb200", "libfluxb200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC,-fvisibility=hidden", "-Xptxas", "-v",
]


def _nvcc() -> str:
    for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if cand and os.path.exists(cand):
            return cand
    raise RuntimeError("nvcc not found")


def _newer(src_paths, target) -> bool:
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in src_paths)


def _fastcall_source(header: str) -> str:
    """C source of the `_fastcall` extension module: one METH_FASTCALL wrapper per entry point of the header that returns
    int32 and takes numbers and single pointers only."""
    text = re.sub(r"/\*.*?\*/", "", open(header).read(), flags=re.S)
    funcs = []
    for m in re.finditer(r"\bint32_t\s+(fb_[a-z0-9_]+)\s*\(([^;]*?)\)\s*;", text, flags=re.S):
        kinds = []
        for a in m.group(2).split(","):
            a = " ".join(a.split())
            stars = a.count("*")
            base = a.replace("const", "").replace("*", "").split()[0]
            if a == "void":
                continue
            kinds.append("?" if stars > 1 else "p" if stars else {"int32_t": "i", "int64_t": "l", "uint64_t": "u", "float": "f"}.get(base, "?"))
        if kinds and "?" not in kinds:
            funcs.append((m.group(1), kinds))
    ctype = {"p": "void*", "i": "int32_t", "l": "int64_t", "u": "uint64_t", "f": "float"}
    out = [open(os.path.join(HERE, "csrc", "fastcall_head.h")).read()]
    for i, (name, kinds) in enumerate(funcs):
        decl = " ".join(f"{ctype[k]} a{j};" for j, k in enumerate(kinds))
        test = " || ".join(f"!get_{k}(a[{j}], &a{j})" for j, k in enumerate(kinds))
        out.append(f"""
static void* fp_{name};
static PyObject* w_{name}(PyObject* self, PyObject* const* a, Py_ssize_t n) {{
  (void)self;
  {decl}
  if (fp_{name} == NULL || n != {len(kinds)} || {test}) Py_RETURN_NONE;
  int32_t r;
  Py_BEGIN_ALLOW_THREADS
  r = ((int32_t (*)({", ".join(ctype[k] for k in kinds)}))fp_{name})({", ".join(f"a{j}" for j in range(len(kinds)))});
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(r);
}}
""")
    out.append("static const struct { const char* name; void** slot; } slots[] = {\n")
    out += [f'  {{"{n}", &fp_{n}}},\n' for n, _ in funcs]
    out.append("  {NULL, NULL}};\nFASTCALL_BIND_AND_NAMES\nstatic PyMethodDef methods[] = {\n")
    out += [f'  {{"{n}", (PyCFunction)(void (*)(void))w_{n}, METH_FASTCALL, NULL}},\n' for n, _ in funcs]
    out.append('  {"bind", do_bind, METH_VARARGS, NULL},\n  {"names", do_names, METH_NOARGS, NULL},\n  {NULL, NULL, 0, NULL}};\nFASTCALL_MODULE\n')
    return "".join(out)


def build_fastcall(force: bool = False):
    """The native call wrappers, generated from the header and compiled with the host compiler.  Optional: without the Python
    headers or a C compiler nothing is built (nor left from an older header), calls go through ctypes, and None is returned."""
    header = os.path.join(HERE, "..", "include", "fluxb200.h")
    head = os.path.join(HERE, "csrc", "fastcall_head.h")
    out = os.path.join(HERE, "fluxb200", "_fastcall" + sysconfig.get_config_var("EXT_SUFFIX"))
    if not force and not _newer([header, head, os.path.abspath(__file__)], out):
        return out
    include, cc = sysconfig.get_paths()["include"], os.environ.get("CC") or "gcc"
    missing = "Python.h" if not os.path.exists(os.path.join(include, "Python.h")) else cc if shutil.which(cc.split()[0]) is None else None
    if missing is not None:
        print(f"no {missing}: the native call wrappers are not built, calls go through ctypes")
        if os.path.exists(out):
            os.remove(out)
        return None
    src = os.path.join(OBJ, "fastcall.c")
    with open(src, "w") as f:
        f.write(_fastcall_source(header))
    cmd = cc.split() + ["-O2", "-shared", "-fPIC", "-I", include, src, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        print(r.stdout + r.stderr)
        raise RuntimeError("building the native call wrappers failed")
    return out


def build(force: bool = False, verbose: bool = False) -> str:
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    sources = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "fluxb200.h"))
    jobs = []
    for s in sources:
        src = os.path.join(CSRC, s)
        obj = os.path.join(OBJ, s[:-3] + ".o")
        if force or _newer([src] + headers, obj):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc] + NVCC_FLAGS + ["-c", src, "-o", obj]
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r.returncode, r.stdout + r.stderr

    log_path = os.path.join(OBJ, "ptxas.log")
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        results = list(ex.map(compile_one, jobs))
    with open(log_path, "a") as log:
        for src, rc, out in results:
            log.write(f"==== {src}\n{out}\n")
            if verbose or rc != 0:
                print(f"==== {src}\n{out}")
            if rc != 0:
                raise RuntimeError(f"nvcc failed on {src}")
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in sources]
    if jobs or force or _newer(objs, OUT):
        cmd = [nvcc, "-shared", "-o", OUT] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            print(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_fastcall(force)
    return OUT


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
