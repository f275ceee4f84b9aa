"""Builds libflashmla_b200.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a.

    python -m flashmla_b200.build [--force] [--verbose]

Each .cu file is compiled to an object (in parallel, skipped when up to date) and the
objects are linked into flashmla_b200/libflashmla_b200.so.  No PyTorch headers are used there.
csrc/host.cpp, the host path of the Python API, is compiled against PyTorch's C++ headers into
flashmla_b200/_host.so.
"""
import argparse
import os
import subprocess
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ_DIR = os.path.join(HERE, "build")
LIB_PATH = os.path.join(HERE, "libflashmla_b200.so")
HOST_PATH = os.path.join(HERE, "_host.so")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "-I", INCLUDE,
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers_mtime():
    deps = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    deps += [os.path.join(INCLUDE, f) for f in os.listdir(INCLUDE)]
    return max(os.path.getmtime(d) for d in deps)


def _compile_one(src, obj, verbose):
    cmd = [_nvcc()] + NVCC_FLAGS + ["-c", src, "-o", obj]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    log = proc.stdout + proc.stderr
    with open(obj + ".log", "w") as f:
        f.write(" ".join(cmd) + "\n" + log)
    if proc.returncode != 0:
        raise RuntimeError(f"nvcc failed for {src}:\n{log}")
    if verbose:
        print(log)
    return log


HOST_LOG = os.path.join(OBJ_DIR, "host.log")          # the command that built the host extension, and what it printed


def _host_command(src):
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(_nvcc())) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    inc = os.path.join(root, "include")
    return [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}", f'-DFLASHMLA_TORCH_VERSION="{torch.__version__}"',
            "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
            "-isystem", sysconfig.get_paths()["include"], "-isystem", os.path.join(cuda, "include"),
            src, "-o", HOST_PATH, "-L" + os.path.join(root, "lib"), "-Wl,-rpath," + os.path.join(root, "lib"),
            "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10", "-lc10_cuda"]


def _host_is_stale(src):
    """Sources newer than the extension, or another command (which names the torch and Python it is compiled against)."""
    newest = max(os.path.getmtime(src), max(os.path.getmtime(os.path.join(INCLUDE, f)) for f in os.listdir(INCLUDE)))
    if not os.path.exists(HOST_PATH) or os.path.getmtime(HOST_PATH) < newest or not os.path.exists(HOST_LOG):
        return True
    with open(HOST_LOG) as f:
        return f.readline().rstrip("\n") != " ".join(_host_command(src))


def _build_host(force):
    src = os.path.join(CSRC, "host.cpp")
    if not force and not _host_is_stale(src):
        return
    cmd = _host_command(src)
    proc = subprocess.run(cmd, capture_output=True, text=True)
    with open(HOST_LOG, "w") as f:
        f.write(("" if proc.returncode == 0 else "failed: ") + " ".join(cmd) + "\n" + proc.stdout + proc.stderr)
    if proc.returncode != 0:
        raise RuntimeError(f"compiling {src} failed:\n" + proc.stdout + proc.stderr)


def build(force=False, verbose=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    hdr_mtime = _headers_mtime()
    jobs = []
    objs = []
    for src in _sources():
        obj = os.path.join(OBJ_DIR, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), hdr_mtime)
        if stale:
            jobs.append((src, obj))
    with ThreadPoolExecutor(max_workers=min(8, len(jobs) + 1)) as ex:
        host = ex.submit(_build_host, force)
        list(ex.map(lambda so: _compile_one(so[0], so[1], verbose), jobs))
        host.result()
    if jobs or not os.path.exists(LIB_PATH):
        cmd = [_nvcc(), "-shared", "-o", LIB_PATH] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-lcudart"]
        proc = subprocess.run(cmd, capture_output=True, text=True)
        if proc.returncode != 0:
            raise RuntimeError("link failed:\n" + proc.stdout + proc.stderr)
    return LIB_PATH


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    args = ap.parse_args()
    print(build(args.force, args.verbose))
