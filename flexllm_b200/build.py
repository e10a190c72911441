"""Builds libflexllm_b200.so (CUDA kernels + C ABI) in-tree with nvcc for sm_100a.

    python -m flexllm_b200.build            # build if sources are newer than the library
    python -m flexllm_b200.build --force
"""
import glob
import os
import subprocess
import sys
import warnings

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "libflexllm_b200.so")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
    # fp32 parity with the reference's C simulation: no fused multiply-add, IEEE div/sqrt, no FTZ
    "-fmad=false", "-prec-div=true", "-prec-sqrt=true", "-ftz=false",
    "-Xcompiler", "-fPIC,-O2,-fvisibility=hidden", "--expt-relaxed-constexpr",
] + os.environ.get("FLEXLLM_NVCC_EXTRA", "").split()      # development aid, e.g. -DFLEXLLM_ATT_TRACE


def gen_exp_constants(path=None):
    """Writes csrc/exp_constants.inc: the constants of the correctly rounded expf kernel helper
    (2^(j/32) table, 32/ln2, ln2/32 split in a short head and a tail), computed here with exact
    integer arithmetic and rounded to double. The generated file is committed; this function is the
    record of how it was made."""
    import math
    from fractions import Fraction

    def to_double(fr):                     # correctly rounded Fraction -> float
        return fr.numerator / fr.denominator   # Python's int/int true division is correctly rounded

    def exp2_frac(j, extra=200):           # 2^(j/32) as a Fraction accurate to ~2^-190
        v = (1 << j) << (32 * extra)
        for _ in range(5):
            v = math.isqrt(v)
        return Fraction(v, 1 << extra)

    ln2 = sum(Fraction(1, k * (1 << k)) for k in range(1, 260))      # ln 2 = sum 1/(k 2^k), error < 2^-260
    c = ln2 / 32
    hi = Fraction(int(c * (1 << 45)), 1 << 45)                       # head: 40 significant bits, so k*head is exact
    lo = c - hi
    lines = ["// Generated by flexllm_b200/build.py:gen_exp_constants(). Do not edit.",
             "// 2^(j/32), j = 0..31, correctly rounded to double",
             "#define FLEXLLM_EXP2_TABLE { \\"]
    for j in range(32):
        lines.append("    %s%s \\" % (to_double(exp2_frac(j)).hex(), "," if j < 31 else ""))
    lines.append("}")
    lines.append("#define FLEXLLM_EXP_INV_LN2_32 %s   // 32 / ln 2" % to_double(32 / ln2).hex())
    lines.append("#define FLEXLLM_EXP_LN2_32_HI %s   // head of ln 2 / 32 (40 bits)" % to_double(hi).hex())
    lines.append("#define FLEXLLM_EXP_LN2_32_LO %s   // tail of ln 2 / 32" % to_double(lo).hex())
    path = path or os.path.join(CSRC, "exp_constants.inc")
    open(path, "w").write("\n".join(lines) + "\n")
    return path


def nccl_include():
    """Directory of nccl.h (the header shipped with torch's NCCL wheel)."""
    try:
        import nvidia
        for p in nvidia.__path__:
            d = os.path.join(p, "nccl", "include")
            if os.path.exists(os.path.join(d, "nccl.h")):
                return d
    except Exception:
        pass
    for d in ("/usr/include", "/usr/local/cuda/include"):
        if os.path.exists(os.path.join(d, "nccl.h")):
            return d
    raise RuntimeError("nccl.h not found")


def nccl_library():
    """Path of libnccl.so.2 next to that header (passed to flexllm_tp_init as a fallback for dlopen)."""
    d = os.path.join(os.path.dirname(nccl_include()), "lib", "libnccl.so.2")
    return d if os.path.exists(d) else "libnccl.so.2"


def sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu")))


def needs_build():
    if not os.path.exists(LIB):
        return True
    t = os.path.getmtime(LIB)
    deps = (sources() + glob.glob(os.path.join(CSRC, "*.cuh")) + glob.glob(os.path.join(CSRC, "*.h")) + glob.glob(os.path.join(CSRC, "*.inc")) +
            glob.glob(os.path.join(HERE, "..", "include", "*.h")))
    return any(os.path.getmtime(d) > t for d in deps)


def front_end_path():
    """File of the Python extension of csrc/front_end.cpp. It is compiled against the layouts of one interpreter and one torch, so its name
    says which: another torch or Python does not find it and gets one of its own."""
    import sysconfig
    import torch
    return os.path.join(HERE, "_front_end.torch-%s%s" % (torch.__version__, sysconfig.get_config_var("EXT_SUFFIX")))


def build_front_end(force=False):
    """Builds that extension (host code against torch's headers)."""
    out = front_end_path()
    src = os.path.join(CSRC, "front_end.cpp")
    header = os.path.join(HERE, "..", "include", "flexllm_b200.h")
    if not force and os.path.exists(out) and os.path.getmtime(out) > max(os.path.getmtime(src), os.path.getmtime(header)):
        return out
    import sysconfig
    import torch
    root = os.path.dirname(torch.__file__)
    cuda = os.path.join(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")), "..", "include")
    part = "%s.%d.part" % (out, os.getpid())                  # never half a file under the name that is loaded
    cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-fvisibility=hidden", "-D_GLIBCXX_USE_CXX11_ABI=%d" % torch._C._GLIBCXX_USE_CXX11_ABI,
           "-I", sysconfig.get_paths()["include"], "-isystem", os.path.join(root, "include"),
           "-isystem", os.path.join(root, "include", "torch", "csrc", "api", "include"), "-I", cuda, src, "-o", part,
           "-L", os.path.join(root, "lib"), "-lc10", "-ltorch_cpu", "-ltorch_python", "-lc10_cuda"]
    try:
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError("g++ failed on front_end.cpp:\n" + r.stdout + r.stderr)
        os.replace(part, out)
    finally:
        if os.path.exists(part):
            os.remove(part)
    return out


def build_library(force=False, verbose=False, ptxas_info=False):
    if not os.path.exists(os.path.join(CSRC, "exp_constants.inc")):
        gen_exp_constants()
    if not force and not needs_build():
        return LIB
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    objs = []
    procs = []
    os.makedirs(os.path.join(HERE, "build"), exist_ok=True)
    for src in sources():
        obj = os.path.join(HERE, "build", os.path.basename(src)[:-3] + ".o")
        objs.append(obj)
        cmd = [nvcc] + NVCC_FLAGS + ["-I", nccl_include()] + (["-Xptxas", "-v"] if ptxas_info else []) + ["-c", src, "-o", obj]
        procs.append((src, subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)))
    log = []
    for src, p in procs:
        out, _ = p.communicate()
        log.append(out)
        if p.returncode != 0:
            raise RuntimeError(f"nvcc failed on {src}:\n{out}")
    cmd = [nvcc, "-shared", "-o", LIB] + objs + ["-gencode", "arch=compute_100a,code=sm_100a"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("link failed:\n" + r.stdout + r.stderr)
    if verbose or ptxas_info:
        print("\n".join(log))
    return LIB


def build(force=False, verbose=False, ptxas_info=False):
    """The library, and the extension where it can be built: without it the calls that it serves take the general path in Python."""
    build_library(force, verbose, ptxas_info)
    try:
        build_front_end(force)
    except (ImportError, OSError, RuntimeError) as e:       # no torch, no compiler, no headers
        warnings.warn("flexllm_b200: the native front end was not built, its calls go through Python: %s" % e)
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, verbose=True, ptxas_info="--ptxas" in sys.argv)
    print("built", LIB)
