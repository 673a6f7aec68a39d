"""Device work of the library runs on the context's stream, which does not wait
for the legacy stream nor hold it up: a clear that goes to the legacy stream is
unordered with the kernels that fill the same buffer."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_clear_on_the_legacy_stream():
    found = []
    for path in glob.glob(os.path.join(ROOT, "cindergs_b200", "csrc", "*.cu*")):
        for k, line in enumerate(open(path), 1):
            if re.search(r"\bcudaMemset(2D)?\(", line.split("//")[0]):
                found.append(f"{os.path.basename(path)}:{k}")
    assert not found, found
