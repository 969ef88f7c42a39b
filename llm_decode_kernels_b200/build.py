"""Build libb200decode.so in-tree with nvcc for sm_100a (no torch headers, no JIT cache), and _host.so, the Python face's native
call path, with the C++ compiler against torch's headers.

    python -m llm_decode_kernels_b200.build [--force] [--verbose]

Each csrc/*.cu is compiled to an object next to the sources (csrc/_obj/) in parallel and linked into
llm_decode_kernels_b200/libb200decode.so. A source is recompiled when it, or any header in csrc/ or include/,
is newer than its object. nvcc cross-compiles without a GPU, so this runs on a CPU-only machine.
"""
import os
import shutil
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor
from pathlib import Path

PKG = Path(__file__).resolve().parent
CSRC = PKG / "csrc"
INCLUDE = PKG.parent / "include"
LIB = PKG / "libb200decode.so"
HOST_SRC = CSRC / "host_ops.cpp"   # the operators' call path, a CPython extension module

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-lineinfo", "-std=c++17",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def nvcc():
    exe = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(exe).exists():
        raise RuntimeError("nvcc not found: libb200decode.so cannot be built on this machine")
    return exe


def sources():
    return sorted(CSRC.glob("*.cu"))


def _newest_header():
    hs = list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.h")) + list(INCLUDE.glob("*.h"))
    return max((h.stat().st_mtime for h in hs), default=0.0)


def build(force=False, verbose=False, defines=(), lib=LIB):
    """Compile what is stale and link. Returns the path of the shared library. `defines` (macro names) and `lib`
    make a variant of the library next to the normal one, with its own object directory: step_trace.py builds
    libb200decode_trace.so with B200_STEP_TRACE this way."""
    lib = Path(lib)
    OBJ = CSRC / ("_obj" if not defines else "_obj_" + "_".join(sorted(defines)).lower())
    OBJ.mkdir(exist_ok=True)
    hdr = _newest_header()
    jobs = []
    for src in sources():
        obj = OBJ / (src.stem + ".o")
        if force or not obj.exists() or obj.stat().st_mtime < max(src.stat().st_mtime, hdr):
            jobs.append((src, obj))

    def compile_one(job):
        src, obj = job
        cmd = [nvcc(), *NVCC_FLAGS, *[f"-D{d}" for d in defines], "-I", str(INCLUDE), "-c", str(src), "-o", str(obj)]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        r = subprocess.run(cmd, capture_output=True, text=True)
        return src, r

    with ThreadPoolExecutor(max_workers=min(8, os.cpu_count() or 1)) as ex:
        for src, r in ex.map(compile_one, jobs):
            if verbose or r.returncode:
                sys.stderr.write(f"--- {src.name}\n{r.stdout}{r.stderr}")
            if r.returncode:
                raise RuntimeError(f"nvcc failed on {src.name}")
    objs = [OBJ / (s.stem + ".o") for s in sources()]
    if jobs or not lib.exists():
        cmd = [nvcc(), "-shared", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(lib), *map(str, objs)]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode:
            sys.stderr.write(r.stdout + r.stderr)
            raise RuntimeError(f"link of {lib.name} failed")
    return lib


def host_path():
    """Where _host lies. The name holds what the module was made for - source, C declarations, torch, Python - so that one made for
    anything else is never loaded."""
    import hashlib
    import sysconfig
    import torch
    h = hashlib.sha256()
    for part in (HOST_SRC.read_bytes(), (INCLUDE / "b200decode.h").read_bytes(), torch.__version__.encode(),
                 sysconfig.get_config_var("SOABI").encode()):
        h.update(part + b"\0")
    return PKG / f"_host_{h.hexdigest()[:16]}.so"


def build_host(force=False, verbose=False):
    """Compile the module of host_path() if it is not there. Returns its path."""
    out = host_path()
    if not force and out.exists():
        return out
    import sysconfig
    import torch
    root = Path(torch.__file__).resolve().parent
    cuda = Path(nvcc()).resolve().parents[1]
    tmp = out.with_name(f".{out.stem}.{os.getpid()}")   # several processes may build at once: each moves a whole file into place
    cmd = [os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
           f"-D_GLIBCXX_USE_CXX11_ABI={int(torch.compiled_with_cxx11_abi())}", "-I", sysconfig.get_paths()["include"],
           "-I", str(root / "include"), "-I", str(root / "include/torch/csrc/api/include"), "-I", str(cuda / "include"),
           str(HOST_SRC), "-o", str(tmp), "-L", str(root / "lib"), "-ltorch_python", "-ltorch_cpu", "-lc10", "-lc10_cuda"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if verbose or r.returncode:
        sys.stderr.write(f"--- {HOST_SRC.name}\n{r.stdout}{r.stderr}")
    if r.returncode:
        tmp.unlink(missing_ok=True)
        raise RuntimeError(f"{cmd[0]} failed on {HOST_SRC.name}")
    os.replace(tmp, out)
    for old in PKG.glob("_host*.so"):
        if old != out:
            old.unlink(missing_ok=True)
    return out


if __name__ == "__main__":
    for step in (build, build_host):
        print(step(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
