"""What the kernels' sources must hold, looked up on the CPU."""
import glob
import os
import re
import subprocess

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "ferrum_b200", "csrc", "kernels")


def test_a_failed_call_is_made_again():
    """An entry point that could not set its kernel up (no device yet, another device) tries again at its next call: no error code is
    kept for the life of the process."""
    kept = [(os.path.basename(f), line) for f in glob.glob(os.path.join(KERNELS, "*.cu*")) for line in open(f)
            if re.search(r"\bstatic\s+(const\s+)?cudaError_t\s+\w+\s*=", line)]
    assert not kept, kept


def test_the_number_of_multiprocessors_is_asked_in_one_place():
    asked = [os.path.basename(f) for f in glob.glob(os.path.join(KERNELS, "*.cu*")) if re.search(r"MultiProcessorCount|multiProcessorCount", open(f).read())]
    assert asked == ["common.cu"], asked


def resources(file, kernel, tmp_path):
    """(bytes of stack, registers) of every instance of a kernel."""
    from ferrum_b200.ops import build
    nvcc = build._find("nvcc", ["/usr/local/cuda/bin"])
    r = subprocess.run([nvcc, *build.NVCC_ARCH, "-O3", "-std=c++17", "-Xptxas", "-v", "-c", os.path.join(KERNELS, file), "-o", str(tmp_path / "o.o")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return [(int(a), int(b)) for a, b in re.findall(
        rf"Compiling entry function '\w*{kernel}\w*'[^\n]*\n(?:[^\n]*Function properties[^\n]*\n)?\s*(\d+) bytes stack frame[^\n]*\n[^\n]*Used (\d+) registers", r.stderr)]


@pytest.mark.parametrize("file,kernel,instances", [("parallel_block.cu", "norm_scaled_add_vec_kernel", 15)])
def test_rows_kept_in_registers_stay_there(file, kernel, instances, tmp_path):
    """Kernels whose comment says that a row stays in registers have no stack."""
    stacks = [n for n, _ in resources(file, kernel, tmp_path)]
    assert len(stacks) == instances and not any(stacks), stacks


def test_half_wide_norms_use_half_the_registers(tmp_path):
    """Rows of two 16-byte pieces a thread are normed in 32 registers, so that eight blocks of 256 threads share an SM."""
    assert max(n for _, n in resources("elementwise.cu", r"rmsnorm_vec_kernel\w*Li2E", tmp_path)) <= 32
