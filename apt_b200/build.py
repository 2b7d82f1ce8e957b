"""Builds apt_b200/libapt_b200.so from apt_b200/csrc/*.cu with nvcc for sm_100a, and apt_b200/_native.so,
the operators' host side in C++ (apt_b200/native/*.cpp), against PyTorch's headers.

Run as ``python apt_b200/build.py`` (add ``--force`` to rebuild, ``-v`` for
ptxas register/shared-memory reports). Run as a file, it does not import the
package, which refuses to load without the library. The library is built
in-tree; nothing is installed.
"""
import os
import shutil
import subprocess
import sys

PKG_DIR = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG_DIR, "csrc")
LIB_PATH = os.path.join(PKG_DIR, "libapt_b200.so")
NATIVE = os.path.join(PKG_DIR, "native")
NATIVE_PATH = os.path.join(PKG_DIR, "_native.so")
SOURCES = ["core.cu", "sample.cu", "relabel.cu", "bucket.cu", "gather.cu", "spmm.cu", "widen.cu", "spmm_f32.cu", "spmm_bf16.cu",
           "spmm_f16.cu", "gat.cu", "virt.cu", "hotness.cu", "p2p.cu", "util.cu"]
NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]


def _nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(exe):
        raise RuntimeError("nvcc not found; libapt_b200.so cannot be built")
    return exe


def _older(target, folder):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    deps = [os.path.join(folder, f) for f in os.listdir(folder)]
    deps.append(os.path.join(PKG_DIR, "..", "include", "apt_b200.h"))
    return any(os.path.getmtime(d) > t for d in deps)


def _native_command(out):
    """g++ on native/*.cpp; PyTorch is found without importing it, its libraries are loaded by the time the
    module is, and libapt_b200.so is the one beside it."""
    import importlib.util
    import sysconfig

    torch_dir = list(importlib.util.find_spec("torch").submodule_search_locations)[0]
    cuda_home = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc())))
    inc = [os.path.join(torch_dir, "include"), os.path.join(torch_dir, "include", "torch", "csrc", "api", "include"),
           os.path.join(cuda_home, "include"), sysconfig.get_paths()["include"]]
    src = sorted(os.path.join(NATIVE, f) for f in os.listdir(NATIVE) if f.endswith(".cpp"))
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-w", "-DTORCH_EXTENSION_NAME=_native",
            *[a for d in inc for a in ("-isystem", d)], *src, "-o", out,
            "-L" + os.path.join(torch_dir, "lib"), "-lc10", "-lc10_cuda", *_cudart(), "-ltorch_cpu", "-ltorch", "-ltorch_python",
            "-Wl,-rpath," + os.path.join(torch_dir, "lib"), "-Wl,-rpath,$ORIGIN", LIB_PATH]


def _cudart():
    """The CUDA runtime PyTorch has loaded: one runtime in the process knows all streams and events."""
    import glob
    import importlib.util

    site = os.path.dirname(list(importlib.util.find_spec("torch").submodule_search_locations)[0])
    found = sorted(glob.glob(os.path.join(site, "nvidia", "*", "lib", "libcudart.so.*")))
    if not found:
        return ["-L" + os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "lib64"), "-lcudart"]
    return [found[0], "-Wl,-rpath," + os.path.dirname(found[0])]


def _build_native(verbose=False):
    tmp_path = NATIVE_PATH + ".tmp"
    subprocess.run(_native_command(tmp_path), check=True)
    os.replace(tmp_path, NATIVE_PATH)


def build(force=False, verbose=False):
    """Compile every kernel file to an object and link the shared library, then the host side over it."""
    if force or _older(LIB_PATH, CSRC):
        _build_kernels(force, verbose)
    if force or _older(NATIVE_PATH, NATIVE):
        _build_native(verbose)
    return LIB_PATH


def _build_kernels(force=False, verbose=False):
    nvcc = _nvcc()
    obj_dir = os.path.join(PKG_DIR, "build")
    os.makedirs(obj_dir, exist_ok=True)
    procs = []
    objs = []
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cuh")]
    headers += [os.path.join(PKG_DIR, "..", "include", "apt_b200.h"), os.path.abspath(__file__)]
    for src in SOURCES:
        obj = os.path.join(obj_dir, src.replace(".cu", ".o"))
        objs.append(obj)
        deps = headers + [os.path.join(CSRC, src)]
        if not force and os.path.exists(obj) and all(os.path.getmtime(d) <= os.path.getmtime(obj) for d in deps):
            continue
        cmd = [nvcc, *NVCC_FLAGS, "-c", os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if p.returncode != 0:
            failed = True
            sys.stderr.write(f"--- nvcc failed on {src}\n{out}\n")
        elif verbose or out.strip():
            sys.stderr.write(f"--- {src}\n{out}\n")
    if failed:
        raise RuntimeError("nvcc failed; see messages above")
    # linked beside its final place and moved there in one step: a reader never sees a half-written library
    tmp_path = LIB_PATH + ".tmp"
    link = [nvcc, "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-Xlinker", "-soname=libapt_b200.so", "-o", tmp_path,
            *objs]
    subprocess.run(link, check=True)
    os.replace(tmp_path, LIB_PATH)


if __name__ == "__main__":
    path = build(force="--force" in sys.argv, verbose="-v" in sys.argv)
    print(path)
