"""Build libb200_hstu.so (the C-ABI library) in-tree with nvcc for sm_100a.

    python generative-recommenders_b200/build.py [--force] [--verbose]

csrc/host.cpp becomes _host.so, the extension module through which the ops queue whole stages.
Each csrc/*.cu becomes build/<name>.o; the objects are linked into
generative-recommenders_b200/libb200_hstu.so.  Files are rebuilt when they or any header
in csrc/ or include/ are newer than their object.
"""

import argparse
import concurrent.futures
import glob
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libb200_hstu.so")
HOST = os.path.join(HERE, "_host.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-lineinfo", "-O3", "-std=c++17",
    "-Xcompiler", "-fPIC",
    "--expt-relaxed-constexpr",
]
# B200_HSTU_TRACE_BUILD=1 compiles the in-kernel timeline marks in (a profiling aid; the marks sit in
# the hot loops, so the default build leaves them out); rebuild with force after changing it
if os.environ.get("B200_HSTU_TRACE_BUILD"):
    NVCC_FLAGS.append("-DB200_HSTU_TRACE_BUILD")


def _nvcc():
    for cand in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", "nvcc"):
        if cand and (os.path.isabs(cand) and os.path.exists(cand) or not os.path.isabs(cand)):
            return cand
    return "nvcc"


def _newest_header():
    hdrs = glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(ROOT, "include", "*.h"))
    return max(os.path.getmtime(h) for h in hdrs)


def _compile(src, obj, verbose):
    cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if verbose else []) + ["-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    return src, r.returncode, r.stdout + r.stderr


def _build_host(force, verbose):
    """csrc/host.cpp -> _host.so, an extension module linked against the library beside it.  It is compiled against
    torch's headers and the interpreter's, so another of either builds it anew (``build/_host.built_with``)."""
    import sysconfig

    import torch

    src, hdr = os.path.join(CSRC, "host.cpp"), os.path.join(ROOT, "include", "b200_hstu.h")
    stamp, built_with = os.path.join(BUILD, "_host.built_with"), "torch %s, python %s" % (torch.__version__, sys.version)
    if (not force and os.path.exists(HOST) and os.path.getmtime(HOST) >= max(os.path.getmtime(src), os.path.getmtime(hdr))
            and os.path.exists(stamp) and open(stamp).read() == built_with):
        return
    t = os.path.dirname(torch.__file__)
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))) if os.path.isabs(_nvcc()) else "/usr/local/cuda"
    includes = [os.path.join(t, "include"), os.path.join(t, "include", "torch", "csrc", "api", "include"),
                sysconfig.get_paths()["include"], os.path.join(cuda, "include")]
    cmd = (["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI]
           + [a for i in includes for a in ("-isystem", i)] + ["-I" + os.path.dirname(hdr), src, "-o", HOST]
           + ["-L" + HERE, "-lb200_hstu", "-L" + os.path.join(t, "lib"), "-lc10", "-lc10_cuda", "-ltorch_cpu", "-ltorch_cuda",
              "-ltorch", "-ltorch_python", "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath,$ORIGIN"])
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0 or verbose:
        sys.stderr.write("== host.cpp (exit %d)\n%s\n" % (r.returncode, r.stdout + r.stderr))
    if r.returncode != 0:
        raise RuntimeError("building _host.so failed")
    with open(stamp, "w") as f:
        f.write(built_with)


def build(force=False, verbose=False):
    os.makedirs(BUILD, exist_ok=True)
    srcs = sorted(glob.glob(os.path.join(CSRC, "*.cu")))
    hdr_time = _newest_header()
    jobs, objs = [], []
    for s in srcs:
        o = os.path.join(BUILD, os.path.splitext(os.path.basename(s))[0] + ".o")
        objs.append(o)
        stale = force or not os.path.exists(o) or os.path.getmtime(o) < max(os.path.getmtime(s), hdr_time)
        if stale:
            jobs.append((s, o))
    failed = False
    with concurrent.futures.ThreadPoolExecutor(max_workers=min(8, max(1, len(jobs)))) as ex:
        for src, rc, out in ex.map(lambda j: _compile(j[0], j[1], verbose), jobs):
            if rc != 0 or verbose:
                sys.stderr.write("== %s (exit %d)\n%s\n" % (os.path.basename(src), rc, out))
            failed = failed or rc != 0
    if failed:
        raise RuntimeError("nvcc failed")
    if jobs or not os.path.exists(LIB):
        cmd = [_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    _build_host(force, verbose)
    return LIB


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--verbose", action="store_true")
    a = ap.parse_args()
    print(build(a.force, a.verbose))
