"""A device with little memory left and no budget (GPU): a path that keeps arrays to save time
gives way to the leaner one. In a child process, whose memory pool holds nothing yet."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = """
import numpy as np
import torch

import vite_b200
from oracle import vite_oracle as vo

rng = np.random.default_rng(1)
n, m = 4_000_000, 100_000
a, b = rng.integers(0, n, m), rng.integers(0, n, m)
a, b = a[a != b], b[a != b]
g = vo._csr_from_list(n, np.concatenate([a, b]), np.concatenate([b, a]), np.ones(2 * len(a)))
want, count = vo.color(g, 8)
hashes = 32 * n  # eight words a vertex
with vite_b200.Context(0) as c:
    c.color(c.generate_rgg(1000), 8)  # the kernel that computes them is loaded
    dev = c.upload(g.rowptr, g.tail, g.weight)
    assert dev.ne >= 1 << 17  # as many entries as make keeping them worth it
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - hashes * 3 // 4, dtype=torch.uint8, device="cuda")
    try:
        c.reserve(hashes)
    except vite_b200.VgError as e:
        assert e.status == vite_b200.VG_ERR_OOM
    else:
        raise AssertionError("the device has room for the hashes")
    got, got_count = c.color(dev, 8)
    assert got_count == count and np.array_equal(got, want)
print("colored")
"""


def test_coloring_without_room_for_its_hashes():
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0 and r.stdout.endswith("colored\n"), r.stderr
