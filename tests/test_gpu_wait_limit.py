"""GPU: the cooperative form's CTAs wait for each other, for about a second at
most.  One that waits for an exchange that nobody comes to (here: its count of
exchanges is put out of step on the host) ends with the timeout status, and
later launches return at once instead of waiting again for numbers that no
longer agree."""
import os
import subprocess

import pytest

from xpbd_gpu import _native

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out(tmp_path):
    exe = str(tmp_path / "gang_wait")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "gang_wait.cu")
    subprocess.run([_native._nvcc(), *_native.ARCH_FLAGS, "-std=c++17", "-O1", src, "-o", exe], check=True, timeout=300)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    rows = [(int(a), float(b), int(c)) for a, b, c in (line.split() for line in out.splitlines())]
    assert [r[0] for r in rows] == [0, 0, 1, 1, 1], out
    assert [r[2] for r in rows] == [5, 10, 10, 10, 10], out  # a CTA that gave up leaves its count
    assert 20.0 < rows[2][1] < 2e4 and max(r[1] for r in rows[3:]) < 5.0, out
