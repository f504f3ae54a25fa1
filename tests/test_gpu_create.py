"""What the first grid of a length costs."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(1, 8192), (2, 2048)])
def test_first_grid_of_a_length_evaluates_few_angles(dim, n):
    """The host evaluates the angles of an octant, not every twiddle of every table: the first
    grid of a length, in a process of its own, takes less than 4 us a point of the axis on
    top of a second one (7 us when each entry was evaluated, a microsecond a sine)."""
    code = ("import time, qsf_gb300 as Q\n"
            "Q.Grid(1, 8, 0.2).close(); Q.Grid(2, 8, 0.2).close()\n"
            "t = []\n"
            "for _ in range(3):\n"
            "    a = time.perf_counter(); g = Q.Grid(%d, %d, 0.3); t.append(time.perf_counter() - a); g.close()\n"
            "print(t[0] - min(t[1:]))\n" % (dim, n))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert float(r.stdout.strip().splitlines()[-1]) < 4e-6 * n
