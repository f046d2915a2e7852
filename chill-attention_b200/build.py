"""Build the CUDA library for sm_100a with nvcc (no other toolchain needed).

    python chill-attention_b200/build.py            # -> chill_attention/_lib/libchill_b200.so

Each mask functor's tensor-core kernels and its CUDA-core kernels are translation units of their own
(csrc/tc_inst.cu, csrc/simt_inst.cu with -DCHILL_INST_MASK=<functor>), compiled in parallel.
``build_library`` is also what ``chill_attention.custom`` calls to produce a private
library for a user-defined mask functor.  The objects of the built-in functors, nine tenths of a build, are kept beside the
library and linked into such private libraries as they are.
"""
from __future__ import annotations

import concurrent.futures as cf
import hashlib
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB_DIR = os.path.join(HERE, "chill_attention", "_lib")
BUILTIN_FUNCTORS = ("FullMask", "CausalMask", "SlidingWindowMask", "ChunkwiseMask", "PrefixLMMask")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC", "-I" + INCLUDE, "-I" + CSRC,
    # several builds of these sources can live in one process (the main library and custom-mask libraries): keep
    # their function-local statics apart instead of merging them as process-wide unique symbols
    "-Xcompiler", "-fno-gnu-unique",
]


def _nvcc():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        raise RuntimeError("nvcc not found")
    return nvcc


def _sources_digest(extra=()):
    h = hashlib.sha256()
    names = sorted(n for n in os.listdir(CSRC) if n != "torch_ext.cpp") + [os.path.join(INCLUDE, "chill_b200.h")]
    for name in names:
        path = name if os.path.isabs(name) else os.path.join(CSRC, name)
        if os.path.isfile(path):
            h.update(os.path.basename(name).encode())  # not the full path: a built tree may be moved
            with open(path, "rb") as f:
                h.update(f.read())
    for e in extra:
        h.update(str(e).encode())
    return h.hexdigest()


def _run(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("command failed: " + " ".join(cmd) + "\n" + r.stdout + r.stderr)
    return r.stdout + r.stderr


def build_library(out_path=None, custom_header=None, custom_functor=None, verbose=False, force=False):
    """Compile and link the library; returns its path.  Skips work when sources are unchanged."""
    out_path = out_path or os.path.join(LIB_DIR, "libchill_b200.so")
    os.makedirs(os.path.dirname(out_path), exist_ok=True)
    # CHILL_B200_NVCC_FLAGS: extra compiler flags, e.g. "-DCHILL_FWD_POLY_NUM=1 -DCHILL_FWD_POLY_DEN=4"
    defines, functors = os.environ.get("CHILL_B200_NVCC_FLAGS", "").split(), list(BUILTIN_FUNCTORS)
    extra = common = tuple(defines)
    if custom_header is not None:
        custom_header = os.path.abspath(custom_header)
        with open(custom_header, "rb") as f:
            extra = extra + (custom_functor, hashlib.sha256(f.read()).hexdigest())
        defines = defines + [f'-DCHILL_CUSTOM_MASK_HEADER="{custom_header}"', f"-DCHILL_CUSTOM_MASK={custom_functor}"]
        functors.append(custom_functor)
    digest = _sources_digest(extra)
    stamp = out_path + ".stamp"
    if not force and os.path.exists(out_path) and os.path.exists(stamp) and open(stamp).read() == digest:
        return out_path
    obj_dir = os.path.join(os.path.dirname(out_path), "obj_" + os.path.basename(out_path))
    kept_dir = os.path.join(LIB_DIR, "obj_builtin_" + _sources_digest(common)[:16])
    for d in (obj_dir, kept_dir):
        os.makedirs(d, exist_ok=True)
    nvcc = [_nvcc()] + (["-Xptxas", "-v"] if verbose else []) + NVCC_FLAGS

    def compile_unit(unit):
        flags, src, obj = unit
        if os.path.dirname(obj) == kept_dir and os.path.exists(obj) and not force:
            return ""
        part = f"{obj}.{os.getpid()}.o"  # a build that is cut off leaves no half-written object under the final name
        out = _run(nvcc + flags + ["-c", os.path.join(CSRC, src), "-o", part])
        os.replace(part, obj)
        return out

    units = [(defines, src + ".cu", os.path.join(obj_dir, src + ".o")) for src in ("chill_abi", "host_pipeline")]
    for fn in functors:
        builtin = fn in BUILTIN_FUNCTORS
        for unit in ("tc", "simt"):
            units.append((list(common if builtin else defines) + [f"-DCHILL_INST_MASK={fn}"], f"{unit}_inst.cu",
                          os.path.join(kept_dir if builtin else obj_dir, f"{unit}_{fn}.o")))
    with cf.ThreadPoolExecutor(max_workers=8) as ex:
        outs = list(ex.map(compile_unit, units))
    if verbose:
        print("\n".join(outs))
    _run([_nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", out_path] + [obj for _, _, obj in units])
    with open(stamp, "w") as f:
        f.write(digest)
    shutil.rmtree(obj_dir, ignore_errors=True)  # not needed once linked
    if custom_header is None:
        for name in os.listdir(LIB_DIR):  # objects of other sources or flags
            if name.startswith("obj_builtin_") and os.path.join(LIB_DIR, name) != kept_dir:
                shutil.rmtree(os.path.join(LIB_DIR, name), ignore_errors=True)
    return out_path


def build_extension(force=False):
    """Compile the native eager-mode call path (csrc/torch_ext.cpp) against the installed torch; returns its path."""
    import sysconfig

    import torch
    from torch.utils.cpp_extension import include_paths, library_paths

    out = os.path.join(LIB_DIR, "_chill_torch.so")
    src = os.path.join(CSRC, "torch_ext.cpp")
    h = hashlib.sha256((torch.__version__ + sys.version).encode())
    for path in (src, os.path.join(INCLUDE, "chill_b200.h")):
        with open(path, "rb") as f:
            h.update(f.read())
    stamp = out + ".stamp"
    if not force and os.path.exists(out) and os.path.exists(stamp) and open(stamp).read() == h.hexdigest():
        return out
    os.makedirs(LIB_DIR, exist_ok=True)
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    includes = include_paths() + [os.path.join(cuda, "include"), sysconfig.get_paths()["include"], INCLUDE]
    _run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
          "-DTORCH_EXTENSION_NAME=_chill_torch"] + [x for i in includes for x in ("-isystem", i)] + [src, "-o", out]
         + [f"-L{p}" for p in library_paths()] + ["-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch", "-ltorch_python"])
    with open(stamp, "w") as f:
        f.write(h.hexdigest())
    return out


if __name__ == "__main__":
    path = build_library(verbose="-v" in sys.argv, force="-f" in sys.argv)
    print(path)
    print(build_extension(force="-f" in sys.argv))
