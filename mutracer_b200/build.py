"""In-tree build of libmutracer_b200.so for sm_100a.

nvcc compiles the device code (-gencode arch=compute_100a,code=sm_100a) and
the host C++ (scene producers, C ABI, context API); the CUDA runtime is linked
statically so the library only needs the driver on the GPU machine.
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
OUT = os.path.join(HERE, "_lib")
LIB = os.path.join(OUT, "libmutracer_b200.so")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
CU = ["megakernel.cu", "pixel_kernels_r128.cu", "pixel_kernels_r255.cu", "batch_noalloc.cu", "wavefront.cu",
      "bvh_build.cu", "blas_refit.cu"]
CPP = ["scene_prep.cpp", "host_api.cpp", "context.cpp", "sizes.cpp", "descriptor.cpp"]
ENERGY_LUT = os.path.join(CSRC, "openpbr_energy_lut.f32")


def _write_energy_lut_source(path):
    """C++ source holding the decoded OpenPBR energy table (Adobe data,
    Apache-2.0) as float32 bit patterns, generated from the committed
    little-endian float32 file."""
    import struct
    raw = open(ENERGY_LUT, "rb").read()
    if len(raw) % 4:
        raise RuntimeError("energy LUT file is not a whole number of float32 values")
    words = struct.unpack("<%dI" % (len(raw) // 4), raw)
    lines = ["// Generated by mutracer_b200/build.py from csrc/openpbr_energy_lut.f32.",
             "// OpenPBR energy-compensation tables: Copyright 2026 Adobe, Apache License 2.0",
             "// (adobe/openpbr-bsdf), as decoded by the reference's decodeOpenPbrEnergyLut.ts.",
             "#include <cstdint>",
             'extern "C" const uint64_t mtp_openpbr_energy_lut_count = %du;' % len(words),
             'extern "C" const uint32_t mtp_openpbr_energy_lut_bits[%d] = {' % len(words)]
    for i in range(0, len(words), 8):
        lines.append("  " + ", ".join("0x%08xu" % w for w in words[i:i + 8]) + ",")
    lines.append("};")
    tmp = path + ".tmp"
    with open(tmp, "w") as f:
        f.write("\n".join(lines) + "\n")
    os.replace(tmp, path)


def _deps():
    files = [os.path.join(CSRC, f) for f in os.listdir(CSRC)]
    files.append(os.path.join(HERE, "..", "include", "mutracer_b200.h"))
    return files


def build(force: bool = False, verbose: bool = False) -> str:
    if not force and os.path.exists(LIB):
        if os.path.getmtime(LIB) >= max(os.path.getmtime(p) for p in _deps()):
            return LIB
    os.makedirs(OUT, exist_ok=True)
    objs = []
    procs = []
    for src in CU:
        obj = os.path.join(OUT, src + ".o")
        cmd = [NVCC, *ARCH, "-lineinfo", "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-c",
               os.path.join(CSRC, src), "-o", obj]
        if verbose:
            cmd.insert(1, "-Xptxas=-v")
        procs.append(subprocess.Popen(cmd))
        objs.append(obj)
    lut_src = os.path.join(OUT, "energy_lut_data.cpp")
    _write_energy_lut_source(lut_src)
    for path in [*(os.path.join(CSRC, c) for c in CPP), lut_src]:
        src = os.path.basename(path)
        obj = os.path.join(OUT, src + ".o")
        cmd = ["g++", "-O2", "-std=c++17", "-fPIC", "-pthread", "-I/usr/local/cuda/include", "-c",
               path, "-o", obj]
        procs.append(subprocess.Popen(cmd))
        objs.append(obj)
    for p in procs:
        if p.wait() != 0:
            raise RuntimeError("compilation failed")
    tmp = LIB + ".tmp"
    subprocess.check_call([NVCC, *ARCH, "-shared", "-cudart", "static", "-o", tmp, *objs,
                           "-Xcompiler", "-pthread"])
    os.replace(tmp, LIB)
    return LIB


if __name__ == "__main__":
    print(build(force="--force" in sys.argv, verbose="-v" in sys.argv))
