"""The committed DRAM figures belong to kernels that exist."""
import json
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "parallel-randomized-cholesky_b200", "csrc")


def test_traffic_entries_name_current_kernels():
    """Every entry that the benchmark reports as traffic says which kernels' bytes
    it sums, and each of them is a kernel of the library."""
    with open(os.path.join(ROOT, "profiles", "dram_traffic.json")) as f:
        traffic = json.load(f)
    kernels = set()
    for name in os.listdir(CSRC):
        if name.endswith(".cu"):
            text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
            kernels |= set(re.findall(r"__global__[^;{]*?(\w+_kernel)\s*\(", text))
    entries = {k for k in traffic if not k.startswith("_")}
    assert set(traffic["_kernels"]) == entries
    for entry, names in traffic["_kernels"].items():
        assert names and set(names) <= kernels, entry
