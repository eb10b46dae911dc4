"""Build the host-emulation library (test infrastructure; g++ only, no GPU, no nvcc)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))


def build_emu(source="emu.cpp", library="libcvb_emu.so", flags=("-O2",)):
    csrc, lib = os.path.join(ROOT, "conversenet_b200", "csrc"), os.path.join(HERE, library)
    srcs = [os.path.join(HERE, source)] + [os.path.join(csrc, f) for f in os.listdir(csrc)
                                               if f.endswith((".cuh", ".h"))]
    if os.path.exists(lib) and all(os.path.getmtime(lib) >= os.path.getmtime(s) for s in srcs):
        return lib
    if not os.path.exists(os.path.join(csrc, "fft_codelets.cuh")):
        from conversenet_b200.build import generate_sources
        generate_sources()
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    cmd = ["g++", *flags, "-std=c++17", "-fPIC", "-shared", "-w", "-ffp-contract=off", "-x", "c++",
           "-I" + cuda_inc, "-o", lib, os.path.join(HERE, source)]
    subprocess.run(cmd, check=True)
    return lib


def build_emu_rp():
    """The real-plane kernels; misaligned accesses trap."""
    return build_emu("emu_rp.cpp", "libcvb_emu_rp.so",
                     ("-O0", "-fsanitize=alignment", "-fsanitize-undefined-trap-on-error"))


if __name__ == "__main__":
    print(build_emu(), build_emu_rp())
