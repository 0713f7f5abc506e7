"""Device memory that the library keeps for twiddles beyond the rings: the natural tables with the first ring
(N = 512 has no others), then at most 32 MB of lane-ordered ones for all lengths, once."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import torch, cuyashe_gb300 as cy
torch.zeros(1, device="cuda")
q = (1 << 62) - 57
def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]
r = cy.Ring(512, q)
start = free()
for _ in range(3):
    for n in (1024, 2048, 4096, 8192, 16384):
        r = cy.Ring(n, q)
    print((start - free()) / 2**20)
"""


def test_lane_tables():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE], cwd=root, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    used = [float(x) for x in out.stdout.split()]
    assert used[0] <= 36  # 32 MB of tables (40 primes), a ring, and the allocator's 2 MB pieces
    assert used[2] <= used[0] + 2
