"""Builds libcutile_b200.so for sm_100a with nvcc (cross-compiles without a GPU) and the host extension _host.so.

Usage: python build.py [--force] [--verbose]
The library is written next to the Python mirror (../cutile_b200/) so that an
in-tree checkout is self-contained.
"""
import importlib.util
import os
import re
import subprocess
import sys
import sysconfig
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
OUT_DIR = os.path.join(os.path.dirname(HERE), "cutile_b200")
LIB = os.path.join(OUT_DIR, "libcutile_b200.so")
HOST = os.path.join(OUT_DIR, "_host.so")  # native call path of the Python package (host.cpp)
OBJ_DIR = os.path.join(HERE, "build")
INCLUDE = os.path.join(os.path.dirname(os.path.dirname(HERE)), "include")

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
         "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-I", INCLUDE]


def sources():
    return sorted(f for f in os.listdir(HERE) if f.endswith(".cu"))


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def build(force=False, verbose=False):
    os.makedirs(OBJ_DIR, exist_ok=True)
    headers = [os.path.join(HERE, f) for f in os.listdir(HERE) if f.endswith((".h", ".cuh"))]
    headers.append(os.path.join(INCLUDE, "cutile_b200.h"))
    jobs, objs = [], []
    for src in sources():
        obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
        objs.append(obj)
        if force or _stale(obj, [os.path.join(HERE, src)] + headers):
            cmd = [NVCC] + FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", os.path.join(HERE, src), "-o", obj]
            jobs.append(cmd)

    def run(cmd):
        r = subprocess.run(cmd, capture_output=True, text=True)
        return cmd, r

    with ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for cmd, r in ex.map(run, jobs):
            if verbose or r.returncode:
                sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
            if r.returncode:
                raise RuntimeError("nvcc failed for " + cmd[-3])
    if jobs or force or _stale(LIB, objs):
        cmd = [NVCC, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a", "-ldl"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError("link failed")
    build_host(force, verbose)
    return LIB


def built_for():
    """What the host extension is compiled against: the torch that is installed (found without importing it) and this
    Python.  None without torch."""
    spec = importlib.util.find_spec("torch")
    if spec is None:
        return None
    torch_dir = os.path.dirname(spec.origin)
    with open(os.path.join(torch_dir, "version.py")) as f:
        version = re.search(r"^__version__ = '([^']*)'", f.read(), re.M).group(1)
    return {"dir": torch_dir, "torch": version, "python": sysconfig.get_config_var("SOABI")}


def build_host(force=False, verbose=False):
    """The CPython extension: compiled against the headers of the torch that imports it, linked to LIB next to it.  Built
    again when its sources, torch or Python have changed.  Without torch there is nothing that could use it."""
    src = os.path.join(HERE, "host.cpp")
    env = built_for()
    if env is None:
        sys.stderr.write("torch is not installed: the host extension of the Python package is not built\n")
        return
    stamp_file, stamp = os.path.join(OBJ_DIR, "host.stamp"), f"{env['torch']} {env['python']}\n"
    same = False
    if os.path.exists(stamp_file):
        with open(stamp_file) as f:
            same = f.read() == stamp
    if same and not (force or _stale(HOST, [src, os.path.join(INCLUDE, "cutile_b200.h")])):
        return
    cuda = os.path.dirname(os.path.dirname(NVCC))
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-D_GLIBCXX_USE_CXX11_ABI=1",
           f'-DCTB_TORCH_VERSION="{env["torch"]}"',
           "-I", sysconfig.get_paths()["include"], "-I", os.path.join(env["dir"], "include"),
           "-I", os.path.join(env["dir"], "include", "torch", "csrc", "api", "include"), "-I", os.path.join(cuda, "include"),
           src, "-o", HOST, "-L", OUT_DIR, "-l:libcutile_b200.so", "-L", os.path.join(env["dir"], "lib"),
           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python", "-Wl,-rpath,$ORIGIN"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(" ".join(cmd) + "\n" + r.stdout + r.stderr)
    if r.returncode:
        raise RuntimeError("the host extension failed to build")
    os.makedirs(OBJ_DIR, exist_ok=True)
    with open(stamp_file, "w") as f:
        f.write(stamp)


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
