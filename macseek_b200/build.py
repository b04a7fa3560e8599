"""In-tree build of libmacseek_b200.so (nvcc, sm_100a).  `python -m macseek_b200.build` or build() from Python."""
import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libmacseek_b200.so")
HOST_SRC = os.path.join(CSRC, "slot_addresses.cpp")
HOST_LIB = os.path.join(HERE, "libmacseek_b200_host.so")    # what reads PyTorch tensors
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-O3", "-std=c++17", "-lineinfo", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-Xptxas", "-v"]


def sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _stale(target, deps):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(d) > t for d in deps)


def _compile(src):
    obj = os.path.join(OBJ, src[:-3] + ".o")
    headers = [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".h"))]
    headers.append(os.path.join(HERE, "..", "include", "macseek_b200.h"))
    if not _stale(obj, [os.path.join(CSRC, src)] + headers):
        return src, 0, ""
    cmd = [NVCC] + ARCH + FLAGS + ["-c", os.path.join(CSRC, src), "-o", obj]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    with open(obj + ".log", "w") as f:
        f.write(r.stdout)
    return src, r.returncode, r.stdout


def _host_stale(target):
    """The sources changed, or another PyTorch or Python is installed than the library was built for (it says which)."""
    if _stale(HOST_LIB, [HOST_SRC, os.path.abspath(__file__)]):
        return True
    with open(HOST_LIB, "rb") as f:
        return target.encode() + b"\0" not in f.read()


def _host_target():
    import torch
    return "torch %s python %d.%d" % (torch.__version__, *sys.version_info[:2])      # as _lib.host_target(), which needs the library


def _build_host():
    target = _host_target()
    if not _host_stale(target):
        return
    import sysconfig
    import torch
    from torch.utils import cpp_extension
    inc = ["-I" + p for p in cpp_extension.include_paths() + [sysconfig.get_paths()["include"]]]
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch.compiled_with_cxx11_abi(),
                           '-DMSB_BUILT_FOR="%s"' % target]
                          + inc + [HOST_SRC, "-o", HOST_LIB, "-L" + lib, "-ltorch_python", "-ltorch_cpu", "-lc10"])


def build(verbose=False, jobs=None):
    os.makedirs(OBJ, exist_ok=True)
    srcs = sources()
    with cf.ThreadPoolExecutor(max_workers=jobs or min(8, len(srcs))) as ex:
        host = ex.submit(_build_host)
        results = list(ex.map(_compile, srcs))
        host.result()
    for src, rc, out in results:
        if rc != 0:
            sys.stderr.write(out)
            raise RuntimeError("nvcc failed on " + src)
        if verbose and out:
            print(out)
    objs = [os.path.join(OBJ, s[:-3] + ".o") for s in srcs]
    if _stale(LIB, objs):
        cmd = [NVCC] + ARCH + ["-shared", "-o", LIB] + objs + ["-lcudart"]
        subprocess.check_call(cmd)
    return LIB


if __name__ == "__main__":
    print(build(verbose="-v" in sys.argv))
