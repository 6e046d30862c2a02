"""Builds the CPU emulator of the register kernel (TEST ONLY): tests/emul/_build/libpado_reg_emul.so."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(os.path.dirname(HERE)), "padeops_b200", "csrc")
OUT = os.path.join(HERE, "_build", "libpado_reg_emul.so")
SRCS = [os.path.join(HERE, "pado_reg_emul.cu")] + [os.path.join(CSRC, f) for f in ("pado_reg_tables.cpp",
                                                                                   "pado_tables.cpp")]
DEPS = SRCS + [os.path.join(CSRC, h) for h in ("pado_reg.cuh", "pado_reg_tables.h", "pado_common.h", "pado_kernels.cuh",
                                               "pado_stream.cuh", "pado_resident.cuh", "pado_tables.h", "pado_once.h")]


def build() -> str:
    if os.path.exists(OUT) and all(os.path.getmtime(OUT) >= os.path.getmtime(d) for d in DEPS):
        return OUT
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-x", "c++", "-O1", "-std=c++17", "-w", "-fPIC", "-shared", f"-I{cuda}/include", "-o", OUT,
                    *SRCS], check=True)
    return OUT
