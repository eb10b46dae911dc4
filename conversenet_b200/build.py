"""Build libconverse_b200.so for sm_100a, in-tree, with plain nvcc.

    python -m conversenet_b200.build [--force] [--ptxas-v]

Steps: regenerate the butterfly codelets, write the registry of compile-time
plans, compile every translation unit in parallel, link one shared library
next to this file.  Nothing here needs a GPU.
"""
import hashlib
import os
import re
import subprocess
import sys
from concurrent.futures import ThreadPoolExecutor

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OBJ = os.path.join(HERE, "build")
LIB = os.path.join(HERE, "libconverse_b200.so")
HOST = os.path.join(HERE, "_host" + (__import__("sysconfig").get_config_var("EXT_SUFFIX") or ".so"))

# Compile-time plans: (RY0, RY1, RX0, RX1, threads, min blocks per SM).
# Padded plane = (RY0*RY1) x (RX0*RX1); radices in the order the planner emits.
STATIC_PLANS = [
    (17, 4, 17, 4, 272, 2),     # 68 x 68    cfg 2 (64+4, scale 2)
    (12, 11, 12, 11, 528, 1),   # 132 x 132  cfg 1 (128+4)
    (17, 8, 17, 8, 544, 1),     # 136 x 136  SRResNet body (128+8)
]

# Compile-time axis plans of the register-FFT multi-pass path: (R0, R1, S0, S1); axis length R0*R1, and
# for a large prime R0 the Rader sub-plan R0-1 = S0*S1 (else 0, 0).  268 = 67 * 4 (ConverseDnCNN) is
# served by the tensor-core multi-pass kernels (GEMM_PLANS) instead.  Reached by full pairs of 264 and 520 planes, and by
# every size through cvb_pair_fwd (bf16 networks: 260 is ConverseDnCNN at 248 x 248).
STRIP2_PLANS = [
    (22, 12, 0, 0),   # 264  SRResNet 256+8
    (20, 13, 0, 0),   # 260  SRResNet up2 256+4
    (26, 20, 0, 0),   # 520  SRResNet 512+8
    (43, 12, 7, 6),   # 516  USRNet blocks 512+4
    (17, 8, 0, 0),    # 136  (cvb_pair_fwd with CVB_OPT_MULTIPASS)
    (17, 4, 0, 0),    # 68   (likewise)
]

# First factor R0 of the tensor-core multi-pass plans (padded length 4 * R0, both axes of a plane):
# 268 (ConverseDnCNN) and 516 (ConverseUSRNet blocks).  Measured slower than the register
# transforms, and therefore not listed: 66 (264), 128 (512), 130 (520).
GEMM_PLANS = [67, 129]

# Widths of the matrix stage (CVB_RP_EACH_WIDTH in cvb_rp.cuh)
MATRIX_WIDTHS = [20, 24, 32, 36, 44, 56, 64]

NVCC_FLAGS = ["-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17",
              "-Xcompiler", "-fPIC"] + os.environ.get("CVB_NVCC_DEFS", "").split()   # e.g. -DCVB_TUNING for tuning builds


def _nvcc():
    return os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _run(cmd):
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        raise RuntimeError("command failed: %s\n%s\n%s" % (" ".join(cmd), r.stdout, r.stderr))
    return r.stdout + r.stderr


def _write_if_changed(path, text):
    if os.path.exists(path) and open(path).read() == text:
        return
    with open(path, "w") as f:
        f.write(text)


def generate_sources():
    gen = subprocess.run([sys.executable, os.path.join(CSRC, "gen_codelets.py")],
                         capture_output=True, text=True, check=True).stdout
    _write_if_changed(os.path.join(CSRC, "fft_codelets.cuh"), gen)
    reg = "// GENERATED by build.py from STATIC_PLANS -- do not edit.\n" + "".join(
        "CVB_STATIC(%d, %d, %d, %d, %d, %d)\n" % p for p in STATIC_PLANS)
    _write_if_changed(os.path.join(CSRC, "static_registry.inc"), reg)
    reg2 = "// GENERATED by build.py from STRIP2_PLANS -- do not edit.\n" + "".join(
        "CVB_STRIP2(%d, %d, %d, %d)\n" % p for p in STRIP2_PLANS)
    _write_if_changed(os.path.join(CSRC, "strip2_registry.inc"), reg2)
    reg3 = "// GENERATED by build.py from GEMM_PLANS -- do not edit.\n" + "".join(
        "CVB_GEMM(%d)\n" % r for r in GEMM_PLANS)
    _write_if_changed(os.path.join(CSRC, "gemm_registry.inc"), reg3)


def _units():
    units = [("converse_b200", "converse_b200.cu", []), ("k_dynamic", "k_dynamic.cu", []),
             ("k_strip", "k_strip.cu", []), ("k_block", "k_block.cu", []), ("k_block_tc", "k_block_tc.cu", []), ("k_block_tc2", "k_block_tc2.cu", []),
             ("k_block_tc3", "k_block_tc3.cu", []), ("k_block_mlp", "k_block_mlp.cu", []), ("k_block_train", "k_block_train.cu", [])]
    units += [("k_rp", "k_rp.cu", []), ("k_rp_rows", "k_rp_rows.cu", []), ("k_rp_bwd", "k_rp_bwd.cu", []), ("k_fix", "k_fix.cu", [])]
    for name, io in (("f32", "float"), ("bf16", "__nv_bfloat16")):
        for unit in ("k_rp_cols", "k_rp_plane"):
            units.append(("%s_%s" % (unit, name), unit + ".cu", ["-DCVB_IO=" + io, "-DCVB_IO_NAME=" + name]))
    for width in MATRIX_WIDTHS:
        units.append(("k_rp_matrix_%d" % width, "k_rp_matrix.cu", ["-DCVB_MP=%d" % width]))
    for (a, b, c, d, nt, mb) in STATIC_PLANS:
        units.append(("k_static_%d_%d_%d_%d_%d_%d" % (a, b, c, d, nt, mb), "k_static.cu",
                      ["-DCVB_RY0=%d" % a, "-DCVB_RY1=%d" % b, "-DCVB_RX0=%d" % c, "-DCVB_RX1=%d" % d,
                       "-DCVB_NT=%d" % nt, "-DCVB_MB=%d" % mb]))
    for (a, b, c, d) in STRIP2_PLANS:
        units.append(("k_strip2_%d_%d" % (a, b), "k_strip2.cu",
                      ["-DCVB_R0=%d" % a, "-DCVB_R1=%d" % b, "-DCVB_S0=%d" % c, "-DCVB_S1=%d" % d]))
    for r in GEMM_PLANS:
        units.append(("k_gemmdft_%d" % r, "k_gemmdft.cu", ["-DCVB_G0=%d" % r]))
    return units


def _sources(path, seen):
    """`path` and everything it includes by a quoted name, recursively."""
    path = os.path.normpath(path)
    if path in seen or not os.path.exists(path):
        return seen
    seen.add(path)
    for name in re.findall(r'^\s*#\s*include\s+"([^"]+)"', open(path).read(), re.M):
        _sources(os.path.join(os.path.dirname(path), name), seen)
    return seen


def _stamp(src, defs):
    h = hashlib.sha1()
    for path in sorted(_sources(os.path.join(CSRC, src), set())):
        h.update(open(path, "rb").read())
    h.update(" ".join(NVCC_FLAGS + defs).encode())
    return h.hexdigest()


def _host_command():
    """g++ command of the native host module (csrc/host.cpp) against the installed torch."""
    import sysconfig
    import torch
    inc = os.path.join(os.path.dirname(torch.__file__), "include")
    lib = os.path.join(os.path.dirname(torch.__file__), "lib")
    cuda = os.path.dirname(os.path.dirname(_nvcc()))
    return ["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-w", "-I" + sysconfig.get_paths()["include"], "-I" + inc,
            "-I" + os.path.join(inc, "torch", "csrc", "api", "include"), "-I" + os.path.join(cuda, "include"),
            "-D_GLIBCXX_USE_CXX11_ABI=%d" % int(torch._C._GLIBCXX_USE_CXX11_ABI),
            os.path.join(CSRC, "host.cpp"), "-o", HOST, "-L" + lib, "-ltorch_python", "-ltorch", "-ltorch_cpu", "-lc10",
            "-lc10_cuda", "-Wl,-rpath," + lib]


def build_host(force=False):
    """The native host module next to this file; rebuilt when its source, the C ABI or torch changed."""
    cmd = _host_command()
    h = hashlib.sha1(" ".join(cmd).encode())
    for path in (os.path.join(CSRC, "host.cpp"), os.path.join(HERE, "..", "include", "converse_b200.h")):
        h.update(open(path, "rb").read())
    stamp = os.path.join(OBJ, "host.stamp")
    if not force and os.path.exists(HOST) and os.path.exists(stamp) and open(stamp).read() == h.hexdigest():
        return
    _run(cmd)
    with open(stamp, "w") as f:
        f.write(h.hexdigest())


def build(force=False, ptxas_v=False, verbose=True):
    generate_sources()
    os.makedirs(OBJ, exist_ok=True)
    units = _units()
    jobs = []
    for name, src, defs in units:
        obj = os.path.join(OBJ, name + ".o")
        stamp_path = obj + ".stamp"
        stamp = _stamp(src, defs)
        fresh = (not force and os.path.exists(obj) and os.path.exists(stamp_path)
                 and open(stamp_path).read() == stamp)
        if not fresh:
            cmd = [_nvcc()] + NVCC_FLAGS + (["-Xptxas", "-v"] if ptxas_v else []) + defs + \
                  ["-c", os.path.join(CSRC, src), "-o", obj]
            jobs.append((name, cmd, stamp_path, stamp))
    logs = {}
    host = ThreadPoolExecutor(max_workers=1)
    host_done = host.submit(build_host, force)
    if jobs:
        with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as ex:
            for (name, cmd, stamp_path, stamp), out in zip(jobs, ex.map(lambda j: _run(j[1]), jobs)):
                logs[name] = out
                with open(stamp_path, "w") as f:
                    f.write(stamp)
    if jobs or force or not os.path.exists(LIB):
        objs = [os.path.join(OBJ, name + ".o") for name, _, _ in units]
        _run([_nvcc(), "-shared", "-o", LIB] + objs + ["-lcudart"])
    host_done.result()
    host.shutdown()
    if verbose:
        for name, out in logs.items():
            if ptxas_v and out.strip():
                print("== %s ==\n%s" % (name, out))
        print("built %s (%d unit(s) recompiled)" % (LIB, len(jobs)))
    return LIB


if __name__ == "__main__":
    build(force="--force" in sys.argv, ptxas_v="--ptxas-v" in sys.argv)
