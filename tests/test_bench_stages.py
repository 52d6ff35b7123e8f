"""The bench line's stages name kernels that exist, and those that can be a step's largest have a measured
DRAM figure."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_stages_are_kernels():
    import sys
    sys.path.insert(0, ROOT)
    import bench
    src = ""
    for p in glob.glob(os.path.join(ROOT, "nans_projekat_gb300", "csrc", "*.cu")):
        with open(p) as f:
            src += f.read()
    kernels = set(re.findall(r"__global__[^;{]*?\b(k_\w+)\s*\(", src))
    for name, key in bench.STAGES:
        assert set(name.split(" + ")) <= kernels, name
        if key not in ("k_epa_medium", "k_epa_large"):
            assert bench.measured_traffic(key) > 0, key
