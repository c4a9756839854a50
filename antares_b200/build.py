"""Builds antares_b200/libantares_b200.so from csrc/*.cu with nvcc for sm_100a, and antares_b200/_fastcall.so, the
Python front end's native part, from csrc/fastcall.cpp with g++ (both in-tree, no JIT cache).

  python -m antares_b200.build [--force] [--verbose]
"""
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libantares_b200.so")
FAST_SRC, FAST = os.path.join(CSRC, "fastcall.cpp"), os.path.join(HERE, "_fastcall.so")

NVCC_FLAGS = ["-O3", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo",
              "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr"]


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def up_to_date():
    if not os.path.exists(LIB):
        return False
    t = os.path.getmtime(LIB)
    deps = sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(HERE, "..", "include", "*.h"))
    return all(os.path.getmtime(d) <= t for d in deps)


def built_for():
    """What _fastcall.so depends on besides its source: it calls into torch's and Python's binary interfaces."""
    import torch
    return "torch %s, python %s" % (torch.__version__, sys.version.split()[0])


def build_fastcall(force=False):
    """Needs torch and g++ with Python's headers; the library itself does not, and operators run without it (_lib.fast)."""
    try:
        import torch
    except ImportError as e:
        sys.stderr.write("antares_b200: _fastcall.so not built (%s)\n" % e)
        return None
    import sysconfig
    note = FAST + ".built_for"
    if not force and os.path.exists(FAST) and os.path.getmtime(FAST_SRC) <= os.path.getmtime(FAST) and os.path.exists(note):
        with open(note) as f:
            if f.read() == built_for():
                return FAST
    root = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden",
                           "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
                           '-DAB200_BUILT_FOR="%s"' % built_for(), "-I" + sysconfig.get_paths()["include"],
                           "-I" + os.path.join(root, "include"), "-I" + os.path.join(root, "include", "torch", "csrc", "api", "include"),
                           "-I" + os.path.join(cuda, "include"), FAST_SRC, "-o", FAST + ".new", "-L" + os.path.join(root, "lib"),
                           "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_python"])
    os.replace(FAST + ".new", FAST)
    with open(note, "w") as f:
        f.write(built_for())
    return FAST


def build(force=False, verbose=False):
    lib = build_library(force, verbose)
    try:
        build_fastcall(force)
    except (OSError, subprocess.CalledProcessError) as e:
        sys.stderr.write("antares_b200: _fastcall.so not built (%s)\n" % e)
    return lib


def build_library(force=False, verbose=False):
    if not force and up_to_date():
        return LIB
    objs = []
    procs = []
    for src in sources():
        obj = src[:-3] + ".o"
        cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
        objs.append(obj)
    failed = False
    for src, p in procs:
        out, _ = p.communicate()
        if verbose or p.returncode != 0:
            sys.stderr.write("== %s ==\n%s\n" % (os.path.basename(src), out))
        failed = failed or p.returncode != 0
    if failed:
        raise RuntimeError("nvcc failed")
    subprocess.check_call([_nvcc(), "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"])
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
