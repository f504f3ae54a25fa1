"""2D steps of lengths without kernels of their own, on each of the longer convolution plans
(1536, 2048, 2560, 3072 and 4096 points; the shorter ones are in test_gpu_line_plans.py)."""
import math

import numpy as np
import pytest

from tests import cases as C
from tests.test_gpu_at_size import _fused_vs_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,gauge", [(700, "length"), (1000, "velocity"), (1000, "length"), (1100, "velocity"),
                                     (1500, "length"), (1872, "velocity"), (2000, "length")])
def test_long_convolution_steps_match_oracle(n, gauge):
    """Tolerance as in test_gpu_line_plans.py: (2 dim log2(n) + 10) eps a step, times 4 for the
    up to 13 terms that the oracle's passes of an odd prime factor add up."""
    import qsf_gb300 as Q
    steps = 2
    pulse = dict(field=0.1, omega=1.1, ncycles=1.0)
    got, ref, psi, opsi = _fused_vs_oracle(2, n, 0.3, 2.0, Q.GAUGE_LENGTH if gauge == "length" else Q.GAUGE_VELOCITY,
                                           steps, pulse, seed=n)
    tol = 4 * steps * (4 * math.log2(n) + 10) * 2.2e-16
    assert C.rel_l2(psi, opsi) < tol
    # the last step's sums over the oracle's psi, added pairwise (the oracle adds one by one)
    x = (np.arange(n) - (n - 1) / 2.0) * 0.3
    one = -2.0 / np.sqrt(x * x + 1.0)
    V = one[:, None] + one + 1.0 / np.sqrt((x[:, None] - x) ** 2 + 1.0)
    rho = np.abs(opsi) ** 2 * 0.3 ** 2
    np.testing.assert_allclose(got[-1, :2], [rho.sum(), (V * rho).sum()], rtol=2 * tol, atol=0)
    np.testing.assert_allclose(got[:, 2:], ref[:, 2:], rtol=0, atol=1e-12 * np.abs(ref[:, 2:]).max())
