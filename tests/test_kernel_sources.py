"""What the kernels' sources must hold, looked up on the CPU."""
import glob
import os
import re

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
