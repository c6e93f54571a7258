"""Host-side rules of the kernel launchers, read from the sources."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shared_memory_limits_are_set_per_device():
    """A kernel's dynamic shared-memory limit belongs to a device: a launcher that remembers having set it once per process fails on a second GPU. So the limit
    is set by allow_smem (a bit per device), behind an array with an entry per device, or at every launch."""
    sets = 0
    for path in sorted(glob.glob(os.path.join(ROOT, "vyomai_b200", "csrc", "*.cu*"))):
        src = open(path).read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", src):
            before = src[max(0, m.start() - 250):m.start()]
            kept = re.search(r"\bstatic\s+(bool|size_t|std::once_flag)\s+\w+(\[\w+\])?\s*[={;]", before)
            assert kept is None or "[dev]" in before, (path, src[m.start():m.start() + 100])
            sets += 1
    assert sets > 0
