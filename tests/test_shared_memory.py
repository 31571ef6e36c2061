"""Dynamic shared memory starts where its declaration says: a plain `extern __shared__ float x[]`
promises 4 bytes, and the static arrays before it (which differ between a kernel's instantiations)
decide the rest. The kernels read theirs in wider words, so every such buffer declares 16."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_dynamic_shared_buffers_declare_their_alignment():
    found = 0
    for path in glob.glob(os.path.join(ROOT, "cuda-pro-cell_gb300", "csrc", "*.cu*")):
        for line in open(path):
            if re.search(r"\bextern\s+__shared__", line):
                found += 1
                assert "__align__(16)" in line, (os.path.basename(path), line.strip())
    assert found >= 4
