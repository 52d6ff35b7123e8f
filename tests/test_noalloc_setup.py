"""The allocation-free solve's set-up, which a host runs at start-up with its first call, names every
kernel of the file. One that it left out would be loaded, into device memory, by the first call that
launches it (CUDA loads kernels lazily), which may be in the middle of a frame."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nans_projekat_gb300", "csrc",
                   "noalloc.cu")


def test_the_first_call_loads_every_kernel():
    with open(SRC) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    kernels = set(re.findall(r"__global__[^;{]*?\b(k_\w+)\s*\(", src))
    setup = re.search(r"kernels\[\]\s*=\s*\{(.*?)\};", src, re.S).group(1)
    launched = set(re.findall(r"\b(k_\w+)\s*<<<", src))
    assert len(kernels) >= 5 and launched == kernels
    assert set(re.findall(r"\bk_\w+", setup)) == kernels
