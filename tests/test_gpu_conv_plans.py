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


@pytest.mark.parametrize("dim,n", [(1, 3), (1, 96), (1, 1021), (1, 1536), (2, 65), (2, 100), (2, 320), (3, 21), (3, 24)])
def test_imaginary_time_with_a_length_gauge_field(dim, n):
    """The x.E factors are real there and change |psi|: the halves do not merge.  Lines and
    passes of built and other lengths, Normalize, E_kin every third step."""
    import qsf_gb300 as Q
    from oracle import oracle as O
    from qsf_gb300.propagator import coupling_schedule
    from tests.test_gpu_at_size import _noise_state
    steps, dt, axis = 7, 0.01, {1: 1, 2: 3, 3: 7}[dim]
    psi0 = _noise_state(dim, n, 0.3, n)
    pulse = dict(field=0.3, omega=1.1, ncycles=1.0)
    og = O.Grid(dim, n, 0.3, nCAP=max(1, n // 10), pot=O.POT_EBERLY, Ncharge=float(dim),
                coupling=O.Coupling(O.GAUGE_LENGTH, [O.Field(axis, [O.Pulse(**pulse)])]))
    og.psi[...] = psi0
    prop = O.Propagator(O.MODE_IM, dt, steps, og, ["norm", "normalize", "epot", "ekin"])
    for _ in range(steps):
        prop.make_step()
        prop.compute_each()
    g = Q.Grid(dim, n, 0.3, nCAP=max(1, n // 10), Ncharge=float(dim), gauge=Q.GAUGE_LENGTH, n_fields=1)
    g.upload(psi0)
    rows = coupling_schedule(Q.Coupling(Q.GAUGE_LENGTH, [Q.Field(axis, [Q.Pulse(**pulse)])]), dt, steps)[0]
    out, done = g.step(Q.MODE_IM, dt, steps, rows, obs=Q.OBS_NORM | Q.OBS_EPOT | Q.OBS_EKIN, normalize=True, ekin_interval=3)
    assert done == steps
    # sqrt(n): the oracle's direct DFT passes of a large prime factor add up to n terms
    tol = steps * (2 * dim * math.log2(n) + 10) * 2.2e-16 * math.sqrt(n)
    assert C.rel_l2(g.download(), og.psi) < tol
    for s, r in enumerate(prop.rows):
        assert out[s, 0] == pytest.approx(r["norm"], rel=4 * tol)
        assert out[s, 1] / out[s, 0] == pytest.approx(r["epot"], rel=4 * tol)
        if (s + 1) % 3 == 0 or s + 1 == steps:
            assert out[s, 2] / out[s, 0] == pytest.approx(r["ekin"], rel=8 * tol)
    g.close()


@pytest.mark.parametrize("dim,n,steps", [(1, 700, 2000), (1, 5003, 2000), (1, 9001, 1500), (2, 260, 300), (2, 371, 200)])
def test_norm_of_a_long_run(dim, n, steps):
    """Convolution plans of 3 2^k and 5 2^k points, whose 1 / M no double holds: its rounding
    must not add up over the steps.  Without an absorber the norm changes by what the tables
    hold: 1 / m rounded to a double, known exactly, and the moduli of the phase factors, whose
    roundings average over the points: together within 2^-53 of that a step."""
    from fractions import Fraction

    import qsf_gb300 as Q
    from tests.test_gpu_at_size import _noise_state
    g = Q.Grid(dim, n, 0.2, nCAP=0, Ncharge=float(dim))
    g.upload(_noise_state(dim, n, 0.2, n, width=0.1))
    g.normalize()
    rows, _ = g.step(Q.MODE_RE, 0.05, steps, obs=Q.OBS_NORM)
    g.close()
    m = n ** dim
    one = 1 << (m.bit_length() - 1)
    known = 2.0 * float(Fraction(one / m) * m / one - 1)
    assert abs((rows[-1, 0] - rows[0, 0]) / (steps - 1) - known) < 2.0 ** -53
