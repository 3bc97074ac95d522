"""Builds libmamba_b200.so and _host.so in-tree.

    python -m mamba_b200._build [--force] [--verbose]

libmamba_b200.so (nvcc, sm_100a) is a C-ABI (include/mamba_b200.h) over the CUDA kernels in mamba_b200/csrc.  It links
the CUDA runtime statically, so loading it needs nothing but the driver.  _host.so (g++, mamba_b200/csrc/host) is the
operators' native call path: a Python extension module over PyTorch's C++ tensors that calls the former.
"""
import os
import subprocess
import sys

PKG = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(PKG, "csrc")
OBJ = os.path.join(CSRC, "build")
LIB = os.path.join(PKG, "libmamba_b200.so")
HOST_SRC = os.path.join(CSRC, "host", "torch_calls.cpp")
HOST = os.path.join(PKG, "_host.so")
HOST_BUILT_FOR = os.path.join(OBJ, "host_built_for.txt")      # host_environment() of the last build of _host.so

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-O3", "-std=c++17", "-lineinfo",
    "-Xcompiler", "-fPIC",
    "-Xptxas", "-v",
    "--expt-relaxed-constexpr", "--extended-lambda",
]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    raise RuntimeError("nvcc not found")


def sources():
    return sorted(os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith(".cu"))


def _headers():
    hs = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    hs.append(os.path.join(os.path.dirname(PKG), "include", "mamba_b200.h"))
    return hs


def host_environment():
    """What _host.so has to have been compiled against: it works on PyTorch's C++ objects, whose layout changes between versions."""
    import torch
    return f"torch {torch.__version__} cxx11abi {int(torch._C._GLIBCXX_USE_CXX11_ABI)} {sys.implementation.cache_tag}"


def host_built_for():
    """host_environment() at the last build of _host.so, or None where that was not recorded."""
    try:
        with open(HOST_BUILT_FOR) as f:
            return f.read().strip()
    except OSError:
        return None


def host_stale(obj, newest_hdr):
    return (not os.path.exists(obj) or not os.path.exists(HOST) or os.path.getmtime(obj) < max(os.path.getmtime(HOST_SRC), newest_hdr)
            or host_built_for() != host_environment())


def _host_command(obj):
    """Compiles the call path against the PyTorch that is installed (its libraries are already loaded when _host.so is imported)."""
    import sysconfig
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    return ["/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++", "-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden",
            f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",
            "-isystem", inc, "-isystem", os.path.join(inc, "torch", "csrc", "api", "include"),
            "-isystem", sysconfig.get_paths()["include"], "-isystem", os.path.join(cuda, "include"), "-c", HOST_SRC, "-o", obj]


def build(force=False, verbose=False):
    """Compile every .cu under csrc/ and link libmamba_b200.so, compile and link _host.so; returns the former's path."""
    os.makedirs(OBJ, exist_ok=True)
    nvcc = _nvcc()
    env = dict(os.environ)
    # the image exports CC/CXX to a wrapper; nvcc needs the system host compiler
    host = ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    newest_hdr = max(os.path.getmtime(h) for h in _headers())
    objs, logs = [], []
    procs = []
    for src in sources():
        obj = os.path.join(OBJ, os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        stale = force or not os.path.exists(obj) or os.path.getmtime(obj) < max(os.path.getmtime(src), newest_hdr)
        if stale:
            cmd = [nvcc, *host, *NVCC_FLAGS, "-c", src, "-o", obj]
            procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env, text=True)))
    host_obj = os.path.join(OBJ, "torch_calls.o")
    host_proc = None
    if force or host_stale(host_obj, newest_hdr):
        host_proc = subprocess.Popen(_host_command(host_obj), stdout=subprocess.PIPE, stderr=subprocess.STDOUT, env=env, text=True)
    for src, p in procs:
        out, _ = p.communicate()
        logs.append((src, out))
        if p.returncode != 0:
            sys.stderr.write(out)
            raise RuntimeError(f"nvcc failed on {src}")
        if verbose:
            sys.stderr.write(out)
    if procs or force or not os.path.exists(LIB):
        cmd = [nvcc, *host, "-shared", "-o", LIB, *objs, "-gencode", "arch=compute_100a,code=sm_100a"]
        subprocess.check_call(cmd, env=env)
    if host_proc is not None:
        out, _ = host_proc.communicate()
        if host_proc.returncode != 0:
            sys.stderr.write(out)
            raise RuntimeError(f"g++ failed on {HOST_SRC}")
        import torch
        libs = ["-L", os.path.join(os.path.dirname(torch.__file__), "lib"), "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda",
                "-lc10"]
        subprocess.check_call([_host_command(host_obj)[0], "-shared", "-Wl,--no-as-needed", "-o", HOST, host_obj, "-L", PKG, "-l:libmamba_b200.so",
                               *libs, "-Wl,-rpath,$ORIGIN"], env=env)
        with open(HOST_BUILT_FOR, "w") as f:
            f.write(host_environment() + "\n")
    if logs:
        with open(os.path.join(OBJ, "ptxas.log"), "w") as f:
            for src, out in logs:
                f.write(f"==== {os.path.basename(src)}\n{out}\n")
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
