"""Memory accesses of kernels, checked by running their source on the CPU (tests/cpp/cuda_on_cpu.h): what the
results on a GPU do not show, such as a block that reads what another one writes."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fastimaging_b200", "csrc")
CPP = os.path.join(ROOT, "tests", "cpp")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read().replace("extern __shared__", "extern").replace("__shared__", "static")


def _run(tmp_path, main, headers):
    for name, text in headers.items():
        (tmp_path / name).write_text('#pragma once\n#include "cuda_on_cpu.h"\n' + text)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-I", str(tmp_path), "-I", CPP, os.path.join(CPP, main), "-o",
                    exe], check=True)
    done = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stdout


def test_axis_passes_keep_to_their_own_cells(tmp_path):
    stub = """
namespace stpgpu {
template <typename R> struct Cplx;
template <> struct Cplx<double> { using T = double2; };
template <> struct Cplx<float> { using T = float2; };
struct PackArgs { void* out; };
inline void pack_scalars(const PackArgs&) {}
}
"""
    _run(tmp_path, "fft_axis_main.cpp", {"imager_kernels.cuh": stub, "fft_kernels.cuh": _source("fft_kernels.cuh")})


def test_label_sums(tmp_path):
    """No sums through a range that is not sorted yet; many labels, small and large."""
    src = _source("sourcefind_kernels.cuh")

    def cut(begin, end):
        i = src.index(begin)
        return src[i:src.index(end, i) + len(end)]

    text = (cut("struct FgSizes {", "};\n") + cut("#define FG_LOOP", "blockDim.x)\n") + cut("constexpr int SEG_BIG", "\n")
            + cut("__device__ __forceinline__ uint32_t seg_at", "\n}\n") + cut("constexpr int kSumWarps", "\n}\n"))
    _run(tmp_path, "label_sums_main.cpp", {"label_sums.cuh": text})
